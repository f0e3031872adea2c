// Static Brandes initialisation over K roots.
//
// Replaces BrandesApproxCaseParallel / BrandesSingleTree
// (src/streamingbc_init.c:60-84, :87-183).  Persistent CTAs take roots from an
// atomic counter.  Per root (k_static):
//   forward   level-synchronous BFS; per level the frontier pushes its sigma into
//             the unvisited neighbours (int64 atomics, exact and
//             order-independent), or the unvisited vertices pull it, whichever
//             scans fewer slots.
//   backward  levels from deepest to 0: delta[x] = sigma[x] * sum over children c
//             of w[c] = (delta[c]+1)/sigma[c], the sum pulled by the parents or
//             pushed by the children, again by slots.
// BC is then a column sum of delta over roots excluding each root itself
// (init.c:175-177), k_bc_colsum.
#include <climits>
#include <mutex>
#include <string>
#include <type_traits>
#include "sbc_gb300.h"
#include "sbc_host.h"
#include "sbc_internal.cuh"

namespace sbc {

struct StaticArgs {
    DevGraph G;
    int64_t nv;
    int nk;
    const int64_t* roots;
    int32_t* dist;
    uint8_t* dist8;
    int64_t* sigma;
    double* delta;
    // per-root state derived from the levels, or null where the caller has none
    uint32_t* dist2;
    int32_t* hist;
    int32_t* roster;
    int32_t* roster_n;
    int32_t* roster_dirty;
    ScratchBase scr;
    int halves;        // static workers per update worker's scratch (1 or 2)
    int third_bits;    // kBits: a third bitmap in shared memory, not in scr.st
    int* work_counter;
    unsigned long long* counters;  // [0] vertices, [1] edges
    const int* list;   // roots to (re)compute, or null for all
    const int* nlist;
    const int* abort;  // when non-null and set, the launch does nothing (inputs failed a device check)
    int asym;          // the adjacency is not symmetric (edge_skew sums not to zero)
    const unsigned long long* asym_dev;  // the same, as a sum in device memory (or null)
};

// Where one root's working set lives.
//   kSmall   the whole row (levels, sigma, child weights, queue) and the three
//            bitmaps in shared memory; results are written out once
//   kBits    rows in HBM, bitmaps in shared memory (the one that only a pull
//            writes in HBM: what shared memory leaves is the L1 cache, which
//            the walks of short lists live on)
//   kOneBits the tested bitmap in shared memory, the other two in HBM
//   kNoBits  all bitmaps in HBM
enum StaticMode { kSmall = 0, kBits = 1, kOneBits = 2, kNoBits = 3 };

constexpr int kSlotLevels = 64;   // levels whose slot counts the backward pass can compare
// A vertex is scanned by one lane up to 8 neighbours, by 4 lanes up to 32, by
// 16 up to 128 (each lane then has 8 at a time in flight), by the warp up to
// kBigDeg, and beyond in segments of kSegSlots that the CTA's warps share out.
// A task none of whose vertices has more than kFewSlots takes a shorter form of
// the one-lane step: deep graphs are bound by the instructions of the few warps
// that have work (a path of 20,000, one root 69.8 -> 59.4 ms).  Not where whole
// rows are in shared memory: the graphs that live there have such tasks on
// their outermost levels alone (ER 1,024 would lose half a percent).
constexpr int kLaneSlots = 8, kFewSlots = 4;
constexpr int kBigDeg = 1024;
constexpr int kSegSlots = 2048;
// The backward pass pushes only into vertices of fewer neighbours than 1/16 of
// the graph's largest number, within these bounds: pushed weights are added one
// after the other, and into one address one at a time, while a pull sums a long
// list with 32 lanes a segment.  Largest error of a dependency against long
// double with pulls of a warp alone | pushes into any vertex | this rule:
//   R-MAT 18, 16 roots       2.9e-15 | 3.6e-14 | 1.9e-15
//   R-MAT 20, 8              2.9e-15 | 4.4e-14 | 2.6e-15
//   Chung-Lu 40k, 64         9.2e-16 | 1.3e-15 | 6.8e-16
//   5 hubs, 100k leaves, 16  1.4e-14 | 1.9e-12 | 9.5e-16
// 1/8 puts R-MAT 18 at 4.1e-15, a lower bound of 256 Chung-Lu 40k at 1.4e-15.
// The time of the two last forms: R-MAT 18, 251 roots 9.4 | 10.7 ms, R-MAT 20,
// 304 roots 44.4 | 46.3 ms, Chung-Lu 40k, 256 roots 1.15 | 1.22 ms (1.30 with a
// lower bound of 64); a star of 5,000, 300 roots 1.41 | 0.18 ms.
constexpr int kPushDegMin = 128, kPushDegMax = 4096, kPushDegPart = 16;
constexpr int kLongShift = 40;
// Vertices of kBigDeg or more listed per walk (the others stay a warp's).
constexpr int kBigCap = 1024, kBigCapSmall = 64;

template <int NT, int CAP>
struct StaticSmem {
    static constexpr int kCap = CAP;
    int item, tail, next, next_seg, nbig;
    int max_deg;
    unsigned long long total;
    unsigned long long slots[2], long_slots[2];  // of the level being listed, by its parity
    unsigned long long lvslots[kSlotLevels];  // of each level's vertices
    unsigned long long lvlong[kSlotLevels];   // of those too long to push into; their number from bit kLongShift on
    int big[CAP];
    int seg_end[CAP];  // running segment counts of big[]
    unsigned char bighit[CAP];
    int buf[NT / 32][64];
    unsigned char order[NT / 32][32];
    int wsum[NT / 32];
    unsigned long long walked_v, walked_e, scanned;
};

__device__ __forceinline__ bool bit_of(const uint32_t* B, int k) { return (B[k >> 5] >> (k & 31)) & 1u; }

// Neighbours s0, s0 + step, ... of a list of d slots at rs (-1 past its end).
template <int S>
__device__ __forceinline__ void load_slots(const DevGraph& G, int64_t rs, int d, int s0, int step, int (&k)[S])
{
#pragma unroll
    for (int u = 0; u < S; ++u) k[u] = s0 + step * u < d ? G.col[rs + s0 + step * u] : -1;
}

// Bit u: k[u] is a neighbour (>= 0) and in bitmap B.  All words are loaded
// before any is tested.
template <int S>
__device__ __forceinline__ unsigned in_bitmap(const uint32_t* B, const int (&k)[S])
{
    unsigned w[S];
#pragma unroll
    for (int u = 0; u < S; ++u) w[u] = B[max(k[u], 0) >> 5];
    unsigned in = 0;
#pragma unroll
    for (int u = 0; u < S; ++u) in |= (k[u] >= 0 ? (w[u] >> (k[u] & 31)) & 1u : 0u) << u;
    return in;
}

// Bit u: k[u] is a neighbour.
template <int S>
__device__ __forceinline__ unsigned present(const int (&k)[S])
{
    unsigned in = 0;
#pragma unroll
    for (int u = 0; u < S; ++u) in |= (k[u] >= 0 ? 1u : 0u) << u;
    return in;
}

// s += val[k[u]] over the k[u] in bitmap B; returns their bits.  Every
// neighbour is tested, then the values are gathered, then summed.
template <class T, int S>
__device__ __forceinline__ unsigned sum_in(const uint32_t* B, const T* val, const int (&k)[S], T& s)
{
    const unsigned in = in_bitmap(B, k);
    T y[S];
#pragma unroll
    for (int u = 0; u < S; ++u) y[u] = (in >> u) & 1u ? val[k[u]] : (T)0;
#pragma unroll
    for (int u = 0; u < S; ++u)
        if ((in >> u) & 1u) s += y[u];
    return in;
}

// Appends k[u] for every set bit u of each calling lane's `first`: the lanes
// here reserve the queue's slots together.
template <class Sm, int S>
__device__ __forceinline__ void append_first(Sm& sm, int32_t* q, const int (&k)[S], unsigned first)
{
    const unsigned act = __activemask();
    if (!__any_sync(act, first)) return;
    const unsigned below = (1u << (threadIdx.x & 31)) - 1u;
    int total = 0, at[S];
#pragma unroll
    for (int u = 0; u < S; ++u) {
        const unsigned m = __ballot_sync(act, (first >> u) & 1u);
        at[u] = total + __popc(m & below);
        total += __popc(m);
    }
    const int leader = __ffs(act) - 1;
    int base = 0;
    if ((int)(threadIdx.x & 31) == leader) base = atomicAdd(&sm.tail, total);
    base = __shfl_sync(act, base, leader);
#pragma unroll
    for (int u = 0; u < S; ++u)
        if ((first >> u) & 1u) q[base + at[u]] = k[u];
}

// *p += v in shared memory, modulo 2^64, as a 32-bit add and a carry: a 64-bit
// shared add is a compare-and-swap loop.
__device__ __forceinline__ void add_shared(int64_t* p, long long v)
{
    const unsigned lo = (unsigned)v;
    const unsigned old = atomicAdd((unsigned*)p, lo);
    const unsigned hi = (unsigned)((unsigned long long)v >> 32) + (old + lo < old ? 1u : 0u);
    if (hi) atomicAdd((unsigned*)p + 1, hi);
}

// A vertex held by one lane of a task: its slots and its value.
template <class V>
struct TaskVertex {
    int x, d;
    int64_t rs;
    V v;
};

// The task's vertices of degree (lo, hi], W lanes each: f(owner lane j or -1,
// rs, d, v, step's first rank) for 32 / W of them at a time, all lanes calling.
template <int W, class Sm, class V, class F>
__device__ __forceinline__ void lane_groups(Sm& sm, const TaskVertex<V>& q, int lo, int hi, F f)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    unsigned char* order = sm.order[threadIdx.x >> 5];
    const bool mine = q.d > lo && q.d <= hi;
    const unsigned m = __ballot_sync(full, mine);
    if (!m) return;
    const int n = __popc(m), rank = __popc(m & ((1u << lane) - 1u));
    if (mine) order[rank] = (unsigned char)lane;
    __syncwarp();
    for (int t = 0; t < n; t += 32 / W) {
        const int at = t + lane / W;
        const int j = at < n ? order[at] : -1;
        const int64_t rj = __shfl_sync(full, q.rs, j & 31);
        const int dj = __shfl_sync(full, q.d, j & 31);
        const V vj = __shfl_sync(full, q.v, j & 31);
        f(j, rj, dj, vj, mine ? rank - t : -1);
    }
    __syncwarp();
}

// One vertex per lane (none where q.d is 0): act(v, k[]) gets the neighbours k
// (-1: none) of a vertex whose value is v, from whichever lane scans them.
// Vertices of degree kBigDeg and more are listed for big_segments.  No block
// barrier inside.
template <bool FEW, class Sm, class V, class Act>
__device__ __forceinline__ void push_batch(const DevGraph& G, Sm& sm, TaskVertex<V> q, Act act)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    if (q.d >= kBigDeg) {
        const int p = atomicAdd(&sm.nbig, 1);
        if (p < Sm::kCap) {
            sm.big[p] = q.x;
            q.d = 0;
        }
    }
    if (FEW && !__any_sync(full, q.d > kFewSlots)) {
        int k[kFewSlots];
        if (q.d > 0) {
            load_slots(G, q.rs, q.d, 0, 1, k);
            act(q.v, k);
        }
        __syncwarp();
        return;
    }
    int k[kLaneSlots];
    if (q.d > 0 && q.d <= kLaneSlots) {
        load_slots(G, q.rs, q.d, 0, 1, k);
        act(q.v, k);
    }
    __syncwarp();
    if (!__any_sync(full, q.d > kLaneSlots)) return;
    lane_groups<4>(sm, q, kLaneSlots, 4 * kLaneSlots, [&](int j, int64_t rj, int dj, V vj, int) {
        if (j >= 0) {
            load_slots(G, rj, dj, lane & 3, 4, k);
            act(vj, k);
        }
        __syncwarp();
    });
    lane_groups<16>(sm, q, 4 * kLaneSlots, 16 * kLaneSlots, [&](int j, int64_t rj, int dj, V vj, int) {
        if (j >= 0) {
            load_slots(G, rj, dj, lane & 15, 16, k);
            act(vj, k);
        }
        __syncwarp();
    });
    for (unsigned m = __ballot_sync(full, q.d > 16 * kLaneSlots); m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        const int64_t rj = __shfl_sync(full, q.rs, j);
        const int dj = __shfl_sync(full, q.d, j);
        const V vj = __shfl_sync(full, q.v, j);
        for (int s0 = lane; s0 < dj; s0 += 32 * kLaneSlots) {
            load_slots(G, rj, dj, s0, 32, k);
            act(vj, k);
        }
        __syncwarp();
    }
}

// One vertex per lane: sums val[k] over the neighbours k in bitmap B, the
// lists shared out as in push_batch, and calls done(x, sum, whether any
// neighbour passed) in the lane that brought x.
template <bool FEW, class T, class Sm, class Done>
__device__ __forceinline__ void pull_batch(const DevGraph& G, Sm& sm, TaskVertex<int> q, bool ok,
                                           const uint32_t* B, const T* val, Done done)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    if (q.d >= kBigDeg) {
        const int p = atomicAdd(&sm.nbig, 1);
        if (p < Sm::kCap) {
            sm.big[p] = q.x;
            sm.bighit[p] = 0;
            q.d = 0;
            ok = false;  // finished after big_segments
        }
    }
    T sum = (T)0;
    bool hit = false;
    if (FEW && !__any_sync(full, q.d > kFewSlots)) {
        int k[kFewSlots];
        if (q.d > 0) {
            load_slots(G, q.rs, q.d, 0, 1, k);
            hit = sum_in(B, val, k, sum) != 0u;
        }
        __syncwarp();
        if (ok) done(q.x, sum, hit);
        __syncwarp();
        return;
    }
    int k[kLaneSlots];
    auto add = [&](T& s, bool& hit) { hit |= sum_in(B, val, k, s) != 0u; };
    if (q.d > 0 && q.d <= kLaneSlots) {
        load_slots(G, q.rs, q.d, 0, 1, k);
        add(sum, hit);
    }
    __syncwarp();
    auto grouped = [&](auto width, int lo, int hi) {
        constexpr int W = decltype(width)::value;
        lane_groups<W>(sm, q, lo, hi, [&](int j, int64_t rj, int dj, int, int ahead) {
            T s = (T)0;
            bool h = false;
            if (j >= 0) {
                load_slots(G, rj, dj, lane & (W - 1), W, k);
                add(s, h);
            }
            const unsigned hits = __ballot_sync(full, h);
            if (hits) {
#pragma unroll
                for (int o = W / 2; o > 0; o >>= 1) s += __shfl_xor_sync(full, s, o);
                // the vertex's own lane takes its group's total
                const T mine = __shfl_sync(full, s, (ahead * W) & 31);
                if (ahead >= 0 && ahead < 32 / W) {
                    sum = mine;
                    hit = (hits >> (ahead * W)) & ((1u << W) - 1u);
                }
            }
        });
    };
    if (__any_sync(full, q.d > kLaneSlots)) {
        grouped(std::integral_constant<int, 4>(), kLaneSlots, 4 * kLaneSlots);
        grouped(std::integral_constant<int, 16>(), 4 * kLaneSlots, 16 * kLaneSlots);
        for (unsigned m = __ballot_sync(full, q.d > 16 * kLaneSlots); m; m &= m - 1) {
            const int j = __ffs(m) - 1;
            const int64_t rj = __shfl_sync(full, q.rs, j);
            const int dj = __shfl_sync(full, q.d, j);
            T s = (T)0;
            bool h = false;
            for (int s0 = lane; s0 < dj; s0 += 32 * kLaneSlots) {
                load_slots(G, rj, dj, s0, 32, k);
                add(s, h);
            }
            if (__any_sync(full, h)) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(full, s, o);
                if (lane == j) {
                    sum = s;
                    hit = true;
                }
            }
        }
    }
    if (ok) done(q.x, sum, hit);
    __syncwarp();
}

// Vertices of a list, handed to the warps in tasks of up to 32 (fewer when the
// list is short, so that more warps have work); batch(task vertex, ok) per
// warp.  The next task's slots and value(x) are loaded before the current one
// is walked.
template <int NT, class V, class Sm, class Value, class Batch>
__device__ __forceinline__ void list_tasks(const DevGraph& G, Sm& sm, const int32_t* list, int n,
                                           unsigned long long slots, Value value, Batch batch)
{
    const int lane = threadIdx.x & 31;
    // a few vertices of short lists are better off in a few warps: each warp
    // that takes part costs a turn of the fp64 pipe and of the queue's counter
    // (grid of 100 x 100, one root 1.78 ms with the level spread over all warps,
    // 1.23 so)
    const int least = slots > 64ull * n ? 1 : slots > 8ull * n ? 4 : 16;
    int t = min(32, max(least, (n + NT / 32 - 1) / (NT / 32)));
    // about kSegSlots * 2 slots a task: lists come in vertex order, which
    // gathers the hubs of some graphs in a few tasks
    if (slots > 64ull * n) t = min(t, max(4, (int)(2ull * kSegSlots * n / slots)));
    // the first tasks go by warp number, the others by claims
    const int given = t * (NT / 32);
    int base = t * (int)(threadIdx.x >> 5);
    auto take = [&](TaskVertex<V>& q, bool& ok) {
        ok = lane < t && base + lane < n;
        q.x = q.d = 0;
        q.rs = 0;
        q.v = (V)0;
        if (ok) {
            q.x = list[base + lane];
            q.rs = G.row[q.x];
            q.d = G.deg[q.x];
            q.v = value(q.x);
        }
        return base < n;
    };
    TaskVertex<V> q;
    bool ok;
    for (bool more = take(q, ok); more;) {
        TaskVertex<V> q2;
        bool ok2 = false;
        more = given < n;
        if (more) {
            if (lane == 0) base = given + atomicAdd(&sm.next, t);
            base = __shfl_sync(0xffffffffu, base, 0);
            more = take(q2, ok2);
        }
        batch(q, ok);
        q = q2;
        ok = ok2;
    }
}

// The walk's listed long vertices, a segment per warp at a time, once every
// task is done: seg(i, x, rs, s0, s1) walks slots [s0, s1) of vertex x =
// big[i].  Called by the whole CTA; returns how many vertices are listed, after
// a block barrier that follows the tasks and, where that is not 0, one that
// follows the segments.
template <class Sm, class Seg>
__device__ __forceinline__ int big_segments(const DevGraph& G, Sm& sm, Seg seg)
{
    __syncthreads();
    const int nb = min(sm.nbig, Sm::kCap);
    if (nb == 0) return 0;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        int run = 0;
        for (int i0 = 0; i0 < nb; i0 += 32) {
            int c = i0 + lane < nb ? (G.deg[sm.big[i0 + lane]] + kSegSlots - 1) / kSegSlots : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(full, c, o);
                if (lane >= o) c += y;
            }
            if (i0 + lane < nb) sm.seg_end[i0 + lane] = run + c;
            run += __shfl_sync(full, c, 31);
        }
        if (lane == 0) sm.next_seg = 0;
    }
    __syncthreads();
    for (;;) {
        int u = 0;
        if (lane == 0) u = atomicAdd(&sm.next_seg, 1);
        u = __shfl_sync(full, u, 0);
        if (u >= sm.seg_end[nb - 1]) break;
        int lo = 0, hi = nb - 1;  // first i with seg_end[i] > u
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (sm.seg_end[mid] > u) hi = mid;
            else lo = mid + 1;
        }
        const int x = sm.big[lo];
        const int d = G.deg[x];
        const int s0 = (u - (lo ? sm.seg_end[lo - 1] : 0)) * kSegSlots;
        seg(lo, x, G.row[x], s0, min(d, s0 + kSegSlots));
    }
    __syncthreads();
    return nb;
}

// The vertices whose bit in V is clear, packed 32 at a time per warp.
template <int NT, class Sm, class Batch>
__device__ __forceinline__ void unset_tasks(const DevGraph& G, Sm& sm, const uint32_t* V, int nw,
                                            Batch batch)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int* buf = sm.buf[threadIdx.x >> 5];
    const int t = min(32, max(1, nw / (NT / 32)));
    int pend = 0, base = 0;
    unsigned mine = 0, have = 0;  // the claimed words, and which lanes' words still have vertices to take
    bool more = true, held = false, ok = false;
    TaskVertex<int> q{0, 0, 0, 0};
    for (;;) {
        while (pend < 32 && (more || have)) {
            if (!have) {
                if (lane == 0) base = atomicAdd(&sm.next, t);
                base = __shfl_sync(full, base, 0);
                more = base < nw;
                mine = more && lane < t && base + lane < nw ? ~V[base + lane] : 0u;
                have = __ballot_sync(full, mine != 0u);
                continue;
            }
            const int j = __ffs(have) - 1;
            have &= have - 1;
            const unsigned w = __shfl_sync(full, mine, j);
            if ((w >> lane) & 1u) buf[pend + __popc(w & ((1u << lane) - 1u))] = (base + j) * 32 + lane;
            pend += __popc(w);
            __syncwarp();
        }
        // the batch's slots are loaded now and walked after the one before it
        const bool ok2 = lane < pend;
        TaskVertex<int> q2{ok2 ? buf[lane] : 0, 0, 0, 0};
        if (ok2) {
            q2.rs = G.row[q2.x];
            q2.d = G.deg[q2.x];
        }
        const int left = max(pend - 32, 0);
        const int rest = lane < left ? buf[32 + lane] : 0;
        __syncwarp();
        if (lane < left) buf[lane] = rest;
        __syncwarp();
        if (held) batch(q, ok);
        if (pend == 0) break;
        pend = left;
        q = q2;
        ok = ok2;
        held = true;
    }
}

// Static Brandes of one root per CTA at a time.
//
// What bounds it: one random 8-byte access per (root, tree edge) and direction
// -- sigma on the way down, the child weight on the way up -- at 32 bytes of
// L2 traffic each; everything else is kept below that.
//   * The level test of a neighbour reads one bit.  A walk only ever asks "is k
//     unvisited / on level l", so the CTA keeps that level (or the visited
//     set) as a bitmap in shared memory (128 KB at 2^20 vertices), where the
//     one-byte distance row cost an L2 sector per scanned slot.
//   * Each pair of levels is walked from its cheaper side: forward, the frontier
//     pushes or, when fewer slots are left, the unvisited vertices pull;
//     backward, the parents pull or, short lists alone (kPushDegMin), the
//     children push.  On R-MAT graphs the hubs sit on the middle levels, and
//     about three times fewer slots are scanned.
//   * Warps take vertices from the level by themselves (list_tasks): two block
//     barriers per level on the way down and three on the way up instead of
//     five per 1,024 vertices, and the counters come from the level sizes
//     instead of shared atomics.
//   * Levels, histogram and rosters leave the kernel with the rows.
template <int NT, int MODE>
__global__ void __launch_bounds__(NT, 1024 / NT) k_static(const __grid_constant__ StaticArgs A)
{
    extern __shared__ __align__(16) unsigned char s_dyn[];
    using Sm = StaticSmem<NT, MODE == kSmall ? kBigCapSmall : kBigCap>;
    __shared__ Sm sm;
    if (A.abort && *A.abort) return;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t nv = A.nv;
    const int nw = (int)((nv + 31) / 32);
    const unsigned nx = (unsigned)nw * 32;  // vertices, up to whole words
    // vertices per thread of a pass over all of them, loads first: with few
    // roots a pass is a chain of load latencies (a 2 M vertex graph, an isolated
    // root 1.97 -> 1.56 ms, 152 roots 3.68 -> 2.58)
    constexpr int kUnroll = MODE == kSmall ? 1 : 4;
    constexpr bool kFew = MODE != kSmall;
    const bool sym = !A.asym && !(A.asym_dev && *A.asym_dev);

    // this worker's queue, level starts, child weights and bitmaps
    const size_t slot = blockIdx.x / A.halves;
    int32_t *qd, *lvl;
    double* acc;
    // the tested bitmap; the visited vertices (isolated ones count as visited);
    // the vertices claimed for the next level, by a push and by a pull (which
    // sets each word from one warp alone and needs no fast bitmap for it)
    uint32_t *B, *V, *Npush, *Npull;
    int32_t* sD = nullptr;
    int64_t* sS = nullptr;
    if (MODE == kSmall) {
        unsigned char* p = s_dyn;
        sS = (int64_t*)p;
        p += 8 * nv;
        acc = (double*)p;
        p += 8 * nv;
        sD = (int32_t*)p;
        p += 4 * nv;
        qd = (int32_t*)p;
        p += 4 * nv;
        lvl = (int32_t*)p;
        p += 4 * nv;
        V = (uint32_t*)p;
        B = V + nw;
        Npush = Npull = B + nw;
    } else {
        const bool second = blockIdx.x % A.halves;
        qd = (second ? A.scr.qa : A.scr.qd) + slot * nv;
        lvl = second ? A.scr.qs + slot * nv : A.scr.lvl + slot * (size_t)(nv + 2);
        acc = (second ? (double*)A.scr.dp : A.scr.acc) + slot * nv;
        if (MODE == kBits) {
            V = (uint32_t*)s_dyn;
            B = Npush = V + nw;
            Npull = A.third_bits ? B + nw : (uint32_t*)(A.scr.st + slot * nv) + (second ? nw : 0);
        } else {
            V = A.scr.bits + slot * bitmap_words(nv);
            Npush = Npull = (uint32_t*)(A.scr.st + slot * nv);
            B = MODE == kOneBits ? (uint32_t*)s_dyn : (uint32_t*)(A.scr.qa + slot * nv);
        }
    }
    if (threadIdx.x == 0) sm.walked_v = sm.walked_e = sm.scanned = 0;
    // the others are kept zero between launches where they are in HBM
    for (int i = threadIdx.x; i < nw; i += NT) {
        B[i] = 0u;
        if (MODE == kSmall || A.third_bits) Npull[i] = 0u;
    }

    for (;;) {
        if (threadIdx.x == 0) {
            sm.item = atomicAdd(A.work_counter, 1);
            sm.total = 0;
            sm.max_deg = 0;
        }
        __syncthreads();
        const int item = sm.item;
        if (item >= (A.list ? *A.nlist : A.nk)) break;
        const int r = A.list ? A.list[item] : item;
        int32_t* gD = A.dist + (size_t)r * nv;
        uint8_t* D8 = A.dist8 + (size_t)r * nv;
        int64_t* gS = A.sigma + (size_t)r * nv;
        double* Dl = A.delta + (size_t)r * nv;
        int32_t* D = MODE == kSmall ? sD : gD;
        int64_t* Sg = MODE == kSmall ? sS : gS;
        const int64_t root64 = A.roots[r];
        // a root outside the graph (only possible through callers whose roots
        // are not checked on the host) keeps an empty tree
        const bool valid = root64 >= 0 && root64 < nv;
        const int root = (int)root64;

        {
            unsigned long long sum = 0;
            int most = 0;
            for (unsigned x0 = threadIdx.x; x0 < nx; x0 += kUnroll * NT) {
                int d[kUnroll];
#pragma unroll
                for (int u = 0; u < kUnroll; ++u) d[u] = x0 + u * NT < nv ? A.G.deg[x0 + u * NT] : 0;
#pragma unroll
                for (int u = 0; u < kUnroll; ++u) {
                    const unsigned x = x0 + u * NT;
                    if (x < nv) {
                        D[x] = SBC_INF;
                        Sg[x] = 0;
                        if (MODE == kSmall) acc[x] = 0.0;
                    }
                    sum += (unsigned)d[u];
                    most = max(most, d[u]);
                    const unsigned word = __ballot_sync(full, x >= nv || (sym && d[u] == 0));
                    if (lane == 0 && x < nx) V[x >> 5] = word;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(full, sum, o);
            if (lane == 0) atomicAdd(&sm.total, sum);
            if (most >= kPushDegMin) atomicMax(&sm.max_deg, most);
        }
        __syncthreads();
        auto push_deg = [&]() { return min(max(sm.max_deg / kPushDegPart, kPushDegMin), kPushDegMax); };
        int nlev = 0, reached = 0;
        unsigned long long visited = 0;
        if (valid) {
            unsigned long long front = (unsigned)A.G.deg[root];
            if (threadIdx.x == 0) {
                D[root] = 0;
                Sg[root] = 1;
                qd[0] = root;
                lvl[0] = 0;
                sm.tail = 1;
                sm.next = sm.nbig = 0;
                sm.slots[1] = sm.long_slots[1] = 0;
                sm.lvslots[0] = front;
                sm.lvlong[0] = (int)front >= push_deg() ? front + (1ull << kLongShift) : 0ull;
                V[root >> 5] |= 1u << (root & 31);
            }
            visited = front;
            // ---- forward: levels 0, 1, ... ----
            int L = 0, lo = 0, hi = 1;
            bool held = false;  // kOneBits: B is a copy of V
            __syncthreads();
            for (;;) {
                const unsigned long long rest = sm.total - visited;
                // the scan for unvisited vertices itself costs about a slot per four vertices
                const bool pull = sym && rest + (unsigned long long)(nv >> 2) < front;
                // a level that may have more vertices than the bitmap has words
                // is listed from N when it is complete, in vertex order
                const bool dense = pull || front >= (unsigned)nw;
                uint32_t* const N = pull ? Npull : Npush;
                if (!pull) {
                    if (threadIdx.x == 0) sm.scanned += front;
                    const uint32_t* T = MODE == kOneBits ? B : V;
                    if (MODE == kOneBits && !held) {
                        for (int i = threadIdx.x; i < nw; i += NT) B[i] = V[i];
                        held = true;
                        __syncthreads();
                    }
                    // An unvisited neighbour gains x's sigma and joins N; where
                    // the level is short its first visitor, the one that sets
                    // the bit, also lists it.
                    auto act = [&](long long s, const auto& k) {
                        constexpr int S = std::extent<std::remove_reference_t<decltype(k)>>::value;
                        const unsigned in = present(k) & ~in_bitmap(T, k);
#pragma unroll
                        for (int u = 0; u < S; ++u)
                            if ((in >> u) & 1u) {
                                if (MODE == kSmall) add_shared(&Sg[k[u]], s);
                                else atomic_add_i64(&Sg[k[u]], s);
                            }
                        unsigned first = in & ~in_bitmap(N, k);
                        if (dense) {
#pragma unroll
                            for (int u = 0; u < S; ++u)
                                if ((first >> u) & 1u) atomicOr(&N[k[u] >> 5], 1u << (k[u] & 31));
                            return;
                        }
                        if (first) {
                            unsigned old[S];
#pragma unroll
                            for (int u = 0; u < S; ++u)
                                old[u] = (first >> u) & 1u ? atomicOr(&N[k[u] >> 5], 1u << (k[u] & 31)) : ~0u;
#pragma unroll
                            for (int u = 0; u < S; ++u) {
                                if ((old[u] >> (k[u] & 31)) & 1u) first &= ~(1u << u);
                                if ((first >> u) & 1u) D[k[u]] = L + 1;
                            }
                        }
                        append_first(sm, qd, k, first);
                    };
                    list_tasks<NT, long long>(A.G, sm, qd + lo, hi - lo, front, [&](int x) { return (long long)Sg[x]; },
                                              [&](const TaskVertex<long long>& q, bool) { push_batch<kFew>(A.G, sm, q, act); });
                    big_segments(A.G, sm, [&](int, int x, int64_t rs, int s0, int s1) {
                        const long long s = Sg[x];
                        for (int i = s0 + lane; i < s1; i += 32 * kLaneSlots) {
                            int k[kLaneSlots];
                            load_slots(A.G, rs, s1, i, 32, k);
                            act(s, k);
                        }
                        __syncwarp();
                    });
                } else {
                    if (threadIdx.x == 0) sm.scanned += rest;
                    if (MODE == kOneBits && held) {
                        for (int i = threadIdx.x; i < nw; i += NT) B[i] = 0u;
                        held = false;
                        __syncthreads();
                    }
                    for (int i = lo + threadIdx.x; i < hi; i += NT) atomicOr(&B[qd[i] >> 5], 1u << (qd[i] & 31));
                    __syncthreads();
                    auto done = [&](int x, int64_t sum, bool hit) {
                        if (hit) Sg[x] = sum;
                        if (hit) atomicOr(&N[x >> 5], 1u << (x & 31));
                    };
                    unset_tasks<NT>(A.G, sm, V, nw, [&](const TaskVertex<int>& q, bool ok) {
                        pull_batch<kFew, int64_t>(A.G, sm, q, ok, B, Sg, done);
                    });
                    const int nb = big_segments(A.G, sm, [&](int b, int x, int64_t rs, int s0, int s1) {
                        int64_t s = 0;
                        unsigned any = 0;
                        for (int i = s0 + lane; i < s1; i += 32 * kLaneSlots) {
                            int k[kLaneSlots];
                            load_slots(A.G, rs, s1, i, 32, k);
                            any |= sum_in(B, Sg, k, s);
                        }
                        if (__any_sync(full, any)) {
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(full, s, o);
                            if (lane == 0) {
                                atomic_add_i64(&Sg[x], s);
                                sm.bighit[b] = 1;
                            }
                        }
                    });
                    if (nb > 0) {
                        for (int b = threadIdx.x; b < nb; b += NT)
                            done(sm.big[b], Sg[sm.big[b]], sm.bighit[b] != 0);
                        __syncthreads();
                    }
                }
                // every thread has read the level's counts; the other buffer
                // holds the next level's
                if (threadIdx.x == 0) {
                    sm.next = sm.nbig = 0;
                    sm.slots[L & 1] = sm.long_slots[L & 1] = 0;
                }
                // B and N are empty again between levels (or B is the visited set)
                if (pull)
                    for (int i = lo + threadIdx.x; i < hi; i += NT) B[qd[i] >> 5] = 0u;
                unsigned long long sum = 0, longs = 0;
                auto count = [&](int x) {
                    const unsigned d = (unsigned)A.G.deg[x];
                    sum += d;
                    if (d >= kPushDegMin && (int)d >= push_deg()) longs += d + (1ull << kLongShift);
                };
                lo = hi;
                if (dense) {
                    // N listed in vertex order, added to the visited set and
                    // emptied: a warp per run of words
                    const int run = ((nw + NT / 32 - 1) / (NT / 32) + 31) & ~31;
                    const int w0 = min(nw, (int)(threadIdx.x >> 5) * run), w1 = min(nw, w0 + run);
                    int c = 0;
                    for (int i = w0 + lane; i < w1; i += 32) c += __popc(N[i]);
                    c = __reduce_add_sync(full, c);
                    if (lane == 0) sm.wsum[threadIdx.x >> 5] = c;
                    __syncthreads();
                    const int mine = lane < NT / 32 ? sm.wsum[lane] : 0;
                    int pos = lo + __reduce_add_sync(full, lane < (int)(threadIdx.x >> 5) ? mine : 0);
                    hi = lo + __reduce_add_sync(full, mine);
                    for (int i0 = w0; i0 < w1 && c; i0 += 32) {
                        const int i = i0 + lane;
                        const unsigned word = i < w1 ? N[i] : 0u;
                        if (word) {
                            N[i] = 0u;
                            V[i] |= word;
                            if (MODE == kOneBits && held) B[i] |= word;
                        }
                        for (unsigned have = __ballot_sync(full, word != 0u); have; have &= have - 1) {
                            const int j = __ffs(have) - 1;
                            const unsigned w = __shfl_sync(full, word, j);
                            if ((w >> lane) & 1u) {
                                const int x = (i0 + j) * 32 + lane;
                                qd[pos + __popc(w & ((1u << lane) - 1u))] = x;
                                D[x] = L + 1;
                                count(x);
                            }
                            pos += __popc(w);
                        }
                    }
                    if (threadIdx.x == 0) sm.tail = hi;
                } else {
                    hi = sm.tail;
                    for (int i = lo + threadIdx.x; i < hi; i += NT) {
                        const int x = qd[i];
                        const unsigned bit = 1u << (x & 31);
                        atomicOr(&V[x >> 5], bit);
                        if (MODE == kOneBits && held) atomicOr(&B[x >> 5], bit);
                        N[x >> 5] = 0u;
                        count(x);
                    }
                }
                if (lo == hi) break;
                ++L;
                if (__any_sync(full, sum != 0)) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(full, sum, o);
                    if (lane == 0) atomicAdd(&sm.slots[L & 1], sum);
                    if (__any_sync(full, longs != 0)) {
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) longs += __shfl_xor_sync(full, longs, o);
                        if (lane == 0) atomicAdd(&sm.long_slots[L & 1], longs);
                    }
                }
                if (threadIdx.x == 0) lvl[L] = lo;
                __syncthreads();
                front = sm.slots[L & 1];
                visited += front;
                if (threadIdx.x == 0 && L < kSlotLevels) {
                    sm.lvslots[L] = front;
                    sm.lvlong[L] = sm.long_slots[L & 1];
                }
            }
            nlev = L + 1;
            reached = hi;

            // ---- backward: each vertex sums its children's weights
            // w = (delta + 1) / sigma, kept in acc ----
            if (MODE == kOneBits && held)
                for (int i = threadIdx.x; i < nw; i += NT) B[i] = 0u;
            auto finish = [&](int x, double sum) {
                const Sigma sw = sigma_of(Sg[x]);
                const double nd = sw.b * sum;
                Dl[x] = nd;
                acc[x] = child_weight(nd + 1.0, sw);
            };
            for (int i = lvl[nlev - 1] + threadIdx.x; i < reached; i += NT) finish(qd[i], 0.0);
            if (threadIdx.x == 0) sm.next = sm.nbig = 0;
            if (nlev > kSlotLevels) {
                // parents below the counted levels are all pulled: the slots of
                // every vertex but those of the counted levels and the last one
                for (int i = lvl[nlev - 1] + threadIdx.x; i < reached; i += NT)
                    atomicAdd(&sm.scanned, 0ull - (unsigned)A.G.deg[qd[i]]);
                if (threadIdx.x < kSlotLevels - 1) atomicAdd(&sm.scanned, 0ull - sm.lvslots[threadIdx.x]);
                if (threadIdx.x == 0) atomicAdd(&sm.scanned, visited);
            }
            __syncthreads();
            int end = reached;  // of level l + 1
            for (int l = nlev - 2; l >= 0; --l) {
                const int a0 = lvl[l], a1 = lvl[l + 1];
                const unsigned long long longs = l < kSlotLevels ? sm.lvlong[l] : 0ull;
                const unsigned long long long_slots = longs & ((1ull << kLongShift) - 1);
                const bool push = sym && l + 1 < kSlotLevels && sm.lvslots[l + 1] + long_slots < sm.lvslots[l];
                const bool part = push && longs != 0;  // long lists are pulled all the same
                if (!push || part) {
                    for (int i = a1 + threadIdx.x; i < end; i += NT) atomicOr(&B[qd[i] >> 5], 1u << (qd[i] & 31));
                    // a few long lists: straight to big_segments
                    const bool listed = part && longs >> kLongShift <= (unsigned)Sm::kCap;
                    if (listed)
                        for (int i = a0 + threadIdx.x; i < a1; i += NT) {
                            const int x = qd[i];
                            if (A.G.deg[x] >= push_deg()) sm.big[atomicAdd(&sm.nbig, 1)] = x;
                        }
                    if (threadIdx.x == 0 && l + 1 < kSlotLevels) sm.scanned += part ? long_slots : sm.lvslots[l];
                    __syncthreads();
                    if (!listed)
                        list_tasks<NT, int>(A.G, sm, qd + a0, a1 - a0, l < kSlotLevels ? sm.lvslots[l] : 0ull,
                                            [](int) { return 0; },
                                            [&](TaskVertex<int> q, bool ok) {
                                                if (part && q.d < push_deg()) {
                                                    q.d = 0;
                                                    ok = false;
                                                }
                                                pull_batch<kFew, double>(A.G, sm, q, ok, B, acc,
                                                                   [&](int y, double sum, bool) { finish(y, sum); });
                                            });
                    const int nb = big_segments(A.G, sm, [&](int, int x, int64_t rs, int s0, int s1) {
                        double s = 0.0;
                        unsigned any = 0;
                        for (int i = s0 + lane; i < s1; i += 32 * kLaneSlots) {
                            int k[kLaneSlots];
                            load_slots(A.G, rs, s1, i, 32, k);
                            any |= sum_in(B, acc, k, s);
                        }
                        if (__any_sync(full, any)) {
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(full, s, o);
                            if (lane == 0) atomicAdd(&acc[x], s);
                        }
                    });
                    if (nb > 0) {
                        for (int b = threadIdx.x; b < nb; b += NT) finish(sm.big[b], acc[sm.big[b]]);
                        __syncthreads();
                    }
                    for (int i = a1 + threadIdx.x; i < end; i += NT) B[qd[i] >> 5] = 0u;
                    if (threadIdx.x == 0) sm.next = sm.nbig = 0;
                    __syncthreads();
                }
                if (push) {
                    for (int i = a0 + threadIdx.x; i < a1; i += NT) {
                        const int x = qd[i];
                        if (!part || A.G.deg[x] < push_deg()) atomicOr(&B[x >> 5], 1u << (x & 31));
                    }
                    if (threadIdx.x == 0) sm.scanned += sm.lvslots[l + 1];
                    __syncthreads();
                    auto act = [&](double w, const auto& k) {
                        constexpr int S = std::extent<std::remove_reference_t<decltype(k)>>::value;
                        const unsigned in = in_bitmap(B, k);
#pragma unroll
                        for (int u = 0; u < S; ++u)
                            if ((in >> u) & 1u) atomicAdd(&acc[k[u]], w);
                    };
                    list_tasks<NT, double>(A.G, sm, qd + a1, end - a1, sm.lvslots[l + 1], [&](int x) { return acc[x]; },
                                           [&](const TaskVertex<double>& q, bool) { push_batch<kFew>(A.G, sm, q, act); });
                    big_segments(A.G, sm, [&](int, int x, int64_t rs, int s0, int s1) {
                        const double w = acc[x];
                        for (int i = s0 + lane; i < s1; i += 32 * kLaneSlots) {
                            int k[kLaneSlots];
                            load_slots(A.G, rs, s1, i, 32, k);
                            act(w, k);
                        }
                        __syncwarp();
                    });
                    for (int i = a0 + threadIdx.x; i < a1; i += NT) {
                        const int x = qd[i];
                        if (bit_of(B, x)) finish(x, acc[x]);
                    }
                    __syncthreads();
                    for (int i = a0 + threadIdx.x; i < a1; i += NT) B[qd[i] >> 5] = 0u;
                    if (threadIdx.x == 0) sm.next = sm.nbig = 0;
                    __syncthreads();
                }
                end = a1;
            }
        }

        // ---- the rows, and what is derived from the levels ----
        uint32_t* D2 = A.dist2 ? A.dist2 + (size_t)r * d2_words(nv) : nullptr;
        for (unsigned x0 = threadIdx.x; x0 < nx; x0 += kUnroll * NT) {
            int d[kUnroll];
            unsigned even[kUnroll], odd[kUnroll];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) d[u] = x0 + u * NT < nv ? D[x0 + u * NT] : SBC_INF;
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                const unsigned x = x0 + u * NT;
                if (x < nv) {
                    D8[x] = enc_d8(d[u]);
                    if (MODE == kSmall) {
                        gD[x] = d[u];
                        gS[x] = Sg[x];
                    } else if (d[u] != SBC_INF) {
                        acc[x] = 0.0;
                    }
                    if (d[u] == SBC_INF) Dl[x] = 0.0;
                }
                const unsigned c = enc_d2(d[u]);
                even[u] = __ballot_sync(full, c & 1u);
                odd[u] = __ballot_sync(full, c & 2u);
                if (MODE >= kOneBits && lane == 0 && x < nx) V[x >> 5] = 0u;
            }
            // two bits per vertex: the ballots of the low and the high bits,
            // spread to even and odd places, half a ballot a lane
            if (D2 && lane < 2 * kUnroll) {
                unsigned e = even[0], o = odd[0];
#pragma unroll
                for (int u = 1; u < kUnroll; ++u)
                    if (lane >> 1 == u) {
                        e = even[u];
                        o = odd[u];
                    }
                auto spread = [](unsigned v) {
                    v &= 0xffffu;
                    v = (v | (v << 8)) & 0x00ff00ffu;
                    v = (v | (v << 4)) & 0x0f0f0f0fu;
                    v = (v | (v << 2)) & 0x33333333u;
                    return (v | (v << 1)) & 0x55555555u;
                };
                const int half = lane & 1;
                const int64_t word = ((int64_t)(x0 - lane + (lane >> 1) * NT) >> 4) + half;
                if (word < d2_words(nv)) D2[word] = spread(e >> (16 * half)) | (spread(o >> (16 * half)) << 1);
            }
        }
        if (A.hist) {
            for (int t = threadIdx.x; t < kHistLevels; t += NT) {
                int n = 0;
                if (t < nlev) n = (t + 1 < nlev && t + 1 < kHistLevels ? lvl[t + 1] : reached) - lvl[t];
                A.hist[(size_t)r * kHistLevels + t] = n;
            }
        }
        if (A.roster) {
            for (int t = 0; t < kRosterLevels; ++t) {
                const size_t at = (size_t)r * kRosterLevels + t;
                const int b0 = t < nlev ? lvl[t] : 0;
                const int n = t < nlev ? (t + 1 < nlev ? lvl[t + 1] : reached) - b0 : 0;
                const bool listed = t >= 2 && n <= kRosterCap;
                if (threadIdx.x == 0) {
                    A.roster_n[at] = listed ? n : kRosterCap + 1;
                    A.roster_dirty[at] = 0;
                }
                if (listed)
                    for (int i = threadIdx.x; i < n; i += NT) A.roster[at * kRosterCap + i] = qd[b0 + i];
            }
        }
        if (threadIdx.x == 0) {
            // the reference counts every reached vertex and its degree in both passes
            sm.walked_v += 2ull * (unsigned)reached;
            sm.walked_e += 2ull * visited;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        atomicAdd(&A.counters[0], sm.walked_v);
        atomicAdd(&A.counters[1], sm.walked_e);
        atomicAdd(&A.counters[4], sm.scanned);
    }
}

// bc[v] = sum over roots r of delta[r][v], skipping v == root.  A block takes
// COLS vertices at a time and shares the roots out among its rows of threads
// (each in root order; the rows are added in order at the end).  Large graphs
// are bound by the fp64 adds (R-MAT 20, 1,024 roots: 2.1 ms, 1.07 G adds at
// about 3 per ns and SM); on small ones the time is the chain of loads per
// thread, so few columns and more rows (ER 1,024, 1,024 roots: 20 us with 32
// columns, 258 us with a thread per vertex).
constexpr int kSumThreads = 512;

template <int COLS>
__global__ void __launch_bounds__(kSumThreads) k_bc_colsum(const double* __restrict__ delta,
                                                           const int64_t* __restrict__ roots, int nk, int64_t nv,
                                                           double* __restrict__ bc, const int* __restrict__ abort)
{
    constexpr int PARTS = kSumThreads / COLS;
    __shared__ double part[PARTS][COLS];
    if (abort && *abort) return;
    const int c = threadIdx.x % COLS, p = threadIdx.x / COLS;
    const int per = (nk + PARTS - 1) / PARTS;
    const int r0 = min(nk, p * per), r1 = min(nk, r0 + per);
    for (int64_t v0 = blockIdx.x * (int64_t)COLS; v0 < nv; v0 += (int64_t)gridDim.x * COLS) {
        const int64_t v = v0 + c;
        double s = 0.0;
        if (v < nv) {
#pragma unroll 8
            for (int r = r0; r < r1; ++r) {
                const double d = delta[(size_t)r * nv + v];
                if (roots[r] != v) s += d;
            }
        }
        part[p][c] = s;
        __syncthreads();
        if (p == 0 && v < nv) {
            for (int q = 1; q < PARTS; ++q) s += part[q][c];
            bc[v] = s;
        }
        __syncthreads();
    }
}

// 32 columns read whole lines; below about 8,192 vertices 8 columns give the
// SMs four times the blocks.
cudaError_t launch_bc_colsum(const double* delta, const int64_t* roots, int nk, int64_t nv, double* bc,
                             const int* abort, cudaStream_t s)
{
    const int cols = nv <= 8192 ? 8 : 32;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((nv + cols - 1) / cols, 8192));
    if (cols == 8) k_bc_colsum<8><<<grid, kSumThreads, 0, s>>>(delta, roots, nk, nv, bc, abort);
    else k_bc_colsum<32><<<grid, kSumThreads, 0, s>>>(delta, roots, nk, nv, bc, abort);
    return cudaGetLastError();
}

// Two-bit rows (dist mod 3, 3 = unreachable; 16 vertices per word) of every
// root, or of the listed roots, from their int32 dist rows.  A thread packs
// one word: 16 consecutive distances, 64 contiguous bytes.
__global__ void k_dist2_rows(const int32_t* __restrict__ dist, int64_t nv, int nk, const int* __restrict__ list,
                             const int* __restrict__ nlist, uint32_t* __restrict__ dist2)
{
    const int64_t nw = d2_words(nv);
    const int64_t rows = list ? *nlist : nk;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < rows * nw;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = list ? list[i / nw] : i / nw;
        const int64_t w = i % nw;
        const int32_t* D = dist + r * nv;
        uint32_t word = 0;
        for (int t = 0; t < 16; ++t) {
            const int64_t k = w * 16 + t;
            word |= (k < nv ? enc_d2(D[k]) : 3u) << (2 * t);
        }
        dist2[r * nw + w] = word;
    }
}

cudaError_t launch_dist2_rows(sbc_forest* f, const int* d_list, const int* d_nlist)
{
    k_dist2_rows<<<f->sm_count * 8, 256, 0, f->g->stream>>>(f->d_dist, f->nv, (int)f->nk, d_list, d_nlist,
                                                             f->d_dist2);
    return cudaGetLastError();
}

namespace {

using StaticKernel = void (*)(StaticArgs);

struct StaticShape {
    int nt, mode, grid, halves;
    size_t dyn;
    StaticKernel kernel;
};

size_t static_dyn(int mode, int64_t nv, bool third)
{
    const size_t nw = (size_t)((nv + 31) / 32) * 4;
    return mode == kSmall ? (size_t)nv * 28 + 3 * nw : mode == kBits ? (third ? 3 : 2) * nw : mode == kOneBits ? nw : 0;
}

template <int CAP>
size_t static_fixed_cap(int nt)
{
    return nt == 128 ? sizeof(StaticSmem<128, CAP>) : nt == 256 ? sizeof(StaticSmem<256, CAP>)
         : nt == 512 ? sizeof(StaticSmem<512, CAP>) : sizeof(StaticSmem<1024, CAP>);
}

size_t static_fixed(int nt, int mode)
{
    return mode == kSmall ? static_fixed_cap<kBigCapSmall>(nt) : static_fixed_cap<kBigCap>(nt);
}

StaticKernel static_kernel(int nt, int mode)
{
    if (mode == kSmall)
        return nt == 128 ? k_static<128, kSmall> : nt == 256 ? k_static<256, kSmall> : k_static<512, kSmall>;
    if (mode == kBits)
        return nt <= 256 ? k_static<256, kBits> : nt == 512 ? k_static<512, kBits> : k_static<1024, kBits>;
    return mode == kOneBits ? k_static<1024, kOneBits> : k_static<1024, kNoBits>;
}

int pow2_floor(int64_t x)
{
    int p = 1;
    while (2ll * p <= x) p *= 2;
    return p;
}

// The launch for nk roots of nv vertices with `workers` scratch slots: the
// first mode whose shared memory one CTA can have, then as many CTAs per SM as
// there are roots for (1,024 threads per SM are shared out among them: the
// kernel takes up to 64 registers per thread), as the shared memory holds and,
// where the rows' scratch is in HBM, as there are scratch slots; an update
// worker's scratch has room for two static workers where the bitmaps are in
// shared memory.  hbm_bits: the scratch has room for bitmaps.
StaticShape static_shape(int64_t nv, int64_t nk, int64_t workers, int sm_count, size_t smem_block, size_t smem_sm,
                         bool hbm_bits)
{
    StaticShape S;
    S.mode = kSmall;
    while (S.mode != kNoBits && static_dyn(S.mode, nv, !hbm_bits) + static_fixed(1024, S.mode) + 1024 > smem_block) ++S.mode;
    S.dyn = static_dyn(S.mode, nv, !hbm_bits);
    S.halves = S.mode == kBits && hbm_bits ? 2 : 1;
    int64_t c = std::max<int64_t>(1, (nk + sm_count - 1) / sm_count);
    c = std::min<int64_t>(c, S.mode == kSmall ? 8 : S.mode == kBits ? 4 : 1);
    if (S.mode != kSmall) c = std::min<int64_t>(c, std::max<int64_t>(1, (workers * S.halves + sm_count - 1) / sm_count));
    // fewer CTAs while the SM's shared memory does not hold them (1 KB each is the system's)
    while (c > 1 && (size_t)c * (S.dyn + static_fixed(pow2_floor(1024 / c), S.mode) + 1024) > smem_sm) --c;
    S.nt = std::max(pow2_floor(1024 / c), S.mode == kSmall ? 128 : S.mode == kBits ? 256 : 1024);
    // A small graph's levels are too short for 1,024 threads (barriers and
    // claims cost more than the extra threads walk): with one CTA per SM,
    // R-MAT 10, 60 roots 100 us with 256 threads, 126 with 1,024; R-MAT 12
    // 187 with 512, 199 with 256, 249 with 1,024.
    if (S.mode == kSmall) S.nt = std::min(S.nt, nv < 2048 ? 256 : 512);
    S.grid = (int)std::min<int64_t>(nk, c * sm_count);
    if (S.mode != kSmall) S.grid = (int)std::min<int64_t>(S.grid, workers * S.halves);
    S.kernel = static_kernel(S.nt, S.mode);
    return S;
}

// The shared-memory limit belongs to the kernel, not to the launch, and host
// threads with graphs of different sizes share it: every call sets the same
// value, all that a CTA of this kernel can have, so that none lowers it between
// another's setting and launch.
cudaError_t static_launch(const StaticShape& S, const StaticArgs& A, size_t smem_block, cudaStream_t s)
{
    if (S.dyn + static_fixed(S.nt, S.mode) > 48 * 1024) {
        const int most = (int)(smem_block - static_fixed(S.nt, S.mode) - 1024);
        cudaError_t e = cudaFuncSetAttribute(S.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e) return e;
    }
    S.kernel<<<S.grid, S.nt, S.dyn, s>>>(A);
    return cudaGetLastError();
}

cudaError_t static_limits(int device, size_t* block, size_t* sm)
{
    int b = 0, m = 0;
    cudaError_t e;
    if ((e = cudaDeviceGetAttribute(&b, cudaDevAttrMaxSharedMemoryPerBlockOptin, device)) ||
        (e = cudaDeviceGetAttribute(&m, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device)))
        return e;
    *block = (size_t)b;
    *sm = (size_t)m;
    return cudaSuccess;
}

}  // namespace

cudaError_t launch_static(sbc_forest* f) { return launch_static_list(f, nullptr, nullptr, f->nk); }

cudaError_t launch_static_list(sbc_forest* f, const int* d_list, const int* d_nlist, int64_t n)
{
    sbc_graph* g = f->g;
    cudaStream_t s = g->stream;
    cudaError_t e;
    size_t smem_block = 0, smem_sm = 0;
    if ((e = static_limits(f->device, &smem_block, &smem_sm))) return e;
    if ((e = cudaMemsetAsync(f->d_counter, 0, sizeof(int), s))) return e;
    StaticArgs A;
    A.G = g->dev();
    A.nv = f->nv;
    A.nk = (int)f->nk;
    A.roots = f->d_roots;
    A.dist = f->d_dist;
    A.dist8 = f->d_dist8;
    A.sigma = f->d_sigma;
    A.delta = f->d_delta;
    A.dist2 = f->d_dist2;
    A.hist = f->d_lvlhist;
    A.roster = f->d_roster;
    A.roster_n = f->d_roster_n;
    A.roster_dirty = f->d_roster_dirty;
    A.scr = f->scratch();
    A.work_counter = f->d_counter;
    A.counters = f->d_counters;
    A.list = d_list;
    A.nlist = d_nlist;
    A.abort = nullptr;
    A.asym = g->edge_skew != 0;
    A.asym_dev = nullptr;
    const StaticShape S = static_shape(f->nv, n, f->workers, f->sm_count, smem_block, smem_sm, true);
    A.halves = S.halves;
    A.third_bits = 0;
    f->prof_begin(PROF_STATIC);
    e = static_launch(S, A, smem_block, s);
    f->prof_end(PROF_STATIC);
    if (e) return e;
    if (d_list) return cudaSuccess;  // the caller moves BC by the listed roots' old and new rows
    return launch_bc_colsum(f->d_delta, f->d_roots, (int)f->nk, f->nv, f->d_bc, nullptr, s);
}

}  // namespace sbc

// ===========================================================================
// Static init without any allocation by the library.
//
// For callers that cannot call cudaMalloc -- code running inside another
// runtime's memory pool, or a host process whose device memory is fully
// reserved up front -- sbc_static_init_noalloc runs the same k_static kernel
// with every byte of its scratch (per-worker queues, level offsets and
// accumulators, the one-byte distance rows, the CSR degrees and the counters)
// carved out of one file-scope device array, g_noalloc_scratch, below.  The
// caller passes the graph and the outputs in its own device memory.  Every GPU
// that loads the library holds this array until the process exits.
// ===========================================================================

namespace sbc {
namespace {

constexpr int64_t kNoallocMaxVertices = SBC_NOALLOC_MAX_VERTICES;
constexpr int64_t kNoallocMaxCells = SBC_NOALLOC_MAX_CELLS;  // roots x vertices
constexpr int kNoallocSlots = SBC_NOALLOC_WORKERS;

constexpr size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
// Layout of the array (byte offsets; each region 256-byte aligned).
constexpr size_t kOffCounters = 0;  // work counter + traversal counters
constexpr size_t kOffDeg = align256(kOffCounters + 16 * sizeof(unsigned long long));
constexpr size_t kOffQd = align256(kOffDeg + sizeof(int32_t) * kNoallocMaxVertices);
constexpr size_t kOffLvl = align256(kOffQd + sizeof(int32_t) * kNoallocSlots * kNoallocMaxVertices);
constexpr size_t kOffAcc = align256(kOffLvl + sizeof(int32_t) * kNoallocSlots * (kNoallocMaxVertices + 2));
constexpr size_t kOffDist8 = align256(kOffAcc + sizeof(double) * kNoallocSlots * kNoallocMaxVertices);
constexpr size_t kNoallocBytes = align256(kOffDist8 + kNoallocMaxCells);
static_assert(kNoallocBytes == SBC_NOALLOC_SCRATCH_BYTES, "scratch size in sbc_gb300.h is out of date");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocBytes];

// Device address of g_noalloc_scratch, looked up once per device.
std::mutex g_noalloc_mu;
void* g_noalloc_ptr[256] = {};

__global__ void k_csr_degrees(const int64_t* __restrict__ off, int64_t nv, int32_t* __restrict__ deg)
{
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < nv; v += (int64_t)gridDim.x * blockDim.x)
        deg[v] = (int32_t)(off[v + 1] - off[v]);
}

// Input check on the device, before k_static touches anything: a root outside
// [0, nv), an offset array that does not start at 0 or decreases, or a
// neighbour id outside [0, nv) sets a bit of *bad (1 roots, 2 offsets, 4
// neighbour ids).  k_static and k_bc_colsum read the word and do nothing when
// it is set, so a bad id never becomes an out-of-bounds access.
// The neighbour ids read are d_col[0 .. d_off[nv]), the caller's CSR.
__global__ void k_noalloc_check(const int64_t* __restrict__ off, const int32_t* __restrict__ col, int64_t nv,
                                const int64_t* __restrict__ roots, int64_t nk, int* __restrict__ bad)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int flags = 0;
    for (int64_t r = t0; r < nk; r += stride)
        if (roots[r] < 0 || roots[r] >= nv) flags |= 1;
    for (int64_t v = t0; v < nv; v += stride)
        if (off[v + 1] < off[v] || (v == 0 && off[0] != 0)) flags |= 2;
    const int64_t ne = off[nv];
    for (int64_t i = t0; i < ne; i += stride) {
        const int32_t c = col[i];
        if (c < 0 || (int64_t)c >= nv) flags |= 4;
    }
    if (flags) atomicOr(bad, flags);
}

// The edge skew (edge_mix summed over all slots) of the caller's CSR, once its
// offsets and ids have passed the check.
__global__ void k_csr_skew(const int64_t* __restrict__ off, const int32_t* __restrict__ col, int64_t nv,
                           const int* __restrict__ bad, unsigned long long* skew)
{
    if (*bad) return;
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    unsigned long long sum = 0;
    for (int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < nv; v += nwarps)
        for (int64_t i = off[v] + lane; i < off[v + 1]; i += 32) sum += edge_mix((int)v, col[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0 && sum) atomicAdd(skew, sum);
}

thread_local std::string t_noalloc_err;

int noalloc_fail(int code, const std::string& msg)
{
    t_noalloc_err = msg;
    return code;
}

// Status of the launch just queued: a launch error names the kernel.
bool noalloc_launch_failed(const char* kernel, int* rc)
{
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) return false;
    *rc = noalloc_fail(SBC_ERR_CUDA, std::string("sbc_static_init_noalloc: ") + kernel + " launch failed: " +
                                         cudaGetErrorString(e));
    return true;
}

}  // namespace

}  // namespace sbc

extern "C" const char* sbc_noalloc_last_error(void) { return sbc::t_noalloc_err.c_str(); }

extern "C" int sbc_static_init_noalloc(int64_t nv, const int64_t* d_off, const int32_t* d_col, int64_t nk,
                                       const int64_t* d_roots, int32_t* d_dist, int64_t* d_sigma, double* d_delta,
                                       double* d_bc, void* stream)
{
    using namespace sbc;
    if (nv < 1 || nk < 1 || !d_off || !d_col || !d_roots || !d_dist || !d_sigma || !d_delta || !d_bc)
        return noalloc_fail(SBC_ERR_ARG, "sbc_static_init_noalloc: null pointer or empty graph/root set");
    if (nv > kNoallocMaxVertices)
        return noalloc_fail(SBC_ERR_ARG, "sbc_static_init_noalloc: more vertices than SBC_NOALLOC_MAX_VERTICES");
    if (nk > nv || nk * nv > kNoallocMaxCells)
        return noalloc_fail(SBC_ERR_ARG,
                            "sbc_static_init_noalloc: roots x vertices exceeds SBC_NOALLOC_MAX_CELLS (or nk > nv)");
    // an error left by earlier work of the caller is reported as such, not
    // as a failure of this call's launches
    const cudaError_t pending = cudaGetLastError();
    if (pending != cudaSuccess)
        return noalloc_fail(SBC_ERR_CUDA, std::string("sbc_static_init_noalloc: CUDA error pending from earlier "
                                                      "work before the call: ") + cudaGetErrorString(pending));
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256)
        return noalloc_fail(SBC_ERR_NOGPU, "sbc_static_init_noalloc: no current CUDA device");
    unsigned char* base = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        if (!g_noalloc_ptr[dev]) {
            void* p = nullptr;
            const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess || !p)
                return noalloc_fail(SBC_ERR_CUDA, std::string("sbc_static_init_noalloc: cudaGetSymbolAddress "
                                                              "failed: ") + cudaGetErrorString(e));
            g_noalloc_ptr[dev] = p;
        }
        base = (unsigned char*)g_noalloc_ptr[dev];
    }
    cudaStream_t s = (cudaStream_t)stream;
    unsigned long long* counters = (unsigned long long*)(base + kOffCounters);
    int* bad = (int*)(counters + 12);
    int32_t* deg = (int32_t*)(base + kOffDeg);
    const int slots = (int)std::min<int64_t>(kNoallocSlots, nk);
    // Clear what must start at zero: the work and traversal counters, the
    // input-check word and the accumulators (a previous call leaves them
    // zero, but a call that failed half-way may not have).
    if (cudaMemsetAsync(counters, 0, 16 * sizeof(unsigned long long), s) != cudaSuccess ||
        cudaMemsetAsync(base + kOffAcc, 0, sizeof(double) * (size_t)slots * (size_t)nv, s) != cudaSuccess)
        return noalloc_fail(SBC_ERR_CUDA, "sbc_static_init_noalloc: clearing scratch failed");
    const int dgrid = (int)std::min<int64_t>((nv + 255) / 256, 4096);
    int rc = SBC_OK;
    k_noalloc_check<<<dgrid, 256, 0, s>>>(d_off, d_col, nv, d_roots, nk, bad);
    if (noalloc_launch_failed("k_noalloc_check", &rc)) return rc;
    k_csr_degrees<<<dgrid, 256, 0, s>>>(d_off, nv, deg);
    if (noalloc_launch_failed("k_csr_degrees", &rc)) return rc;

    k_csr_skew<<<dgrid, 256, 0, s>>>(d_off, d_col, nv, bad, counters + 9);
    if (noalloc_launch_failed("k_csr_skew", &rc)) return rc;

    StaticArgs A;
    A.G.nv = nv;
    A.G.row = d_off;
    A.G.deg = deg;   // plain CSR: every slot is visible (deg0 == deg)
    A.G.deg0 = deg;
    A.G.nsort = deg;
    A.G.col = d_col;
    A.G.seq = d_col;  // never read when deg0 == deg
    A.nv = nv;
    A.nk = (int)nk;
    A.roots = d_roots;
    A.dist = d_dist;
    A.dist8 = base + kOffDist8;
    A.sigma = d_sigma;
    A.delta = d_delta;
    A.dist2 = nullptr;
    A.hist = A.roster = A.roster_n = A.roster_dirty = nullptr;
    // k_static uses only the queue, level-offset and accumulator slots here
    // (its bitmaps fit in shared memory up to kNoallocMaxVertices); the others
    // point at valid (unused) memory.
    A.scr.st = (int32_t*)(base + kOffQd);
    A.scr.dp = (int64_t*)(base + kOffAcc);
    A.scr.qa = (int32_t*)(base + kOffQd);
    A.scr.qs = (int32_t*)(base + kOffQd);
    A.scr.bits = (uint32_t*)(base + kOffQd);
    A.scr.qd = (int32_t*)(base + kOffQd);
    A.scr.lvl = (int32_t*)(base + kOffLvl);
    A.scr.acc = (double*)(base + kOffAcc);
    A.work_counter = (int*)(counters + 8);
    A.counters = counters;
    A.list = nullptr;
    A.nlist = nullptr;
    A.abort = bad;
    A.asym = 0;
    A.asym_dev = counters + 9;
    size_t smem_block = 0, smem_sm = 0;
    if (static_limits(dev, &smem_block, &smem_sm) != cudaSuccess)
        return noalloc_fail(SBC_ERR_CUDA, "sbc_static_init_noalloc: device limits not readable");
    // one CTA per scratch slot
    const StaticShape S = static_shape(nv, slots, slots, slots, smem_block, smem_sm, false);
    if (S.mode > kBits) return noalloc_fail(SBC_ERR_CUDA, "sbc_static_init_noalloc: too little shared memory");
    A.halves = 1;
    A.third_bits = S.mode == kBits;
    if (static_launch(S, A, smem_block, s) != cudaSuccess)
        return noalloc_fail(SBC_ERR_CUDA, "sbc_static_init_noalloc: k_static launch failed");
    if (launch_bc_colsum(d_delta, d_roots, (int)nk, nv, d_bc, bad, s) != cudaSuccess)
        return noalloc_fail(SBC_ERR_CUDA, "sbc_static_init_noalloc: k_bc_colsum launch failed");
    // wait for the work and read the input-check word (a 4-byte copy into a
    // stack variable: no allocation)
    int h_bad = 0;
    cudaError_t e = cudaMemcpyAsync(&h_bad, bad, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess)
        return noalloc_fail(SBC_ERR_CUDA, std::string("sbc_static_init_noalloc: ") + cudaGetErrorString(e));
    if (h_bad) {
        std::string m = "sbc_static_init_noalloc: inputs rejected on the device (outputs not written):";
        if (h_bad & 1) m += " a root outside [0, nv);";
        if (h_bad & 2) m += " d_off not a CSR offset array (d_off[0] != 0 or decreasing);";
        if (h_bad & 4) m += " a neighbour id outside [0, nv);";
        return noalloc_fail(SBC_ERR_ARG, m);
    }
    return SBC_OK;
}
