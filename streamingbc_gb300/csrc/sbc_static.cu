// Static Brandes initialisation over K roots.
//
// Replaces BrandesApproxCaseParallel / BrandesSingleTree
// (src/streamingbc_init.c:60-84, :87-183).  One persistent CTA per worker slot
// takes roots from an atomic counter.  Per root:
//   forward   level-synchronous BFS; a frontier vertex pushes its sigma into
//             every neighbour on the next level (int64 atomics, so the sum is
//             exact and order-independent); the first visitor of a vertex
//             claims it with a CAS on dist and appends it to the next frontier.
//   backward  levels from deepest to 0, pull form: a vertex x sums
//             w[c] = (delta[c]+1)/sigma[c] over its children c (dist[c] =
//             dist[x]+1) and sets delta[x] = sigma[x] * sum; no global atomics.
// BC is then a column sum of delta over roots excluding each root itself
// (init.c:175-177), computed by k_bc_colsum in root order.
#include <climits>
#include <mutex>
#include <string>
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
    int* work_counter;
    unsigned long long* counters;  // [0] vertices, [1] edges
    const int* list;   // roots to (re)compute, or null for all
    const int* nlist;
    const int* abort;  // when non-null and set, the launch does nothing (inputs failed a device check)
    int asym;          // the adjacency is not symmetric (edge_skew sums not to zero)
    const unsigned long long* asym_dev;  // the same, as a sum in device memory (or null)
};

// Where one root's working set lives.
//   kSmall   the whole row (levels, sigma, child weights, queue) and both
//            bitmaps in shared memory; results are written out once
//   kBits    rows in HBM, both bitmaps in shared memory
//   kOneBits the tested bitmap in shared memory, the visited one in HBM
//   kNoBits  both bitmaps in HBM
enum StaticMode { kSmall = 0, kBits = 1, kOneBits = 2, kNoBits = 3 };

constexpr int kSlotLevels = 64;   // levels whose slot counts the backward pass can compare
constexpr int kThreadDeg = 4;     // up to this degree a vertex is one thread's work,
constexpr int kGroupDeg = 64;     // up to this eight lanes',
constexpr int kBigDeg = 16384;    // up to this a warp's, and the CTA's beyond
constexpr int kBigCap = 64;       // CTA-wide vertices listed per walk (the others stay a warp's)

template <int NT>
struct StaticSmem {
    int item, tail, next, nbig;
    unsigned long long slots, total;
    unsigned long long lvslots[kSlotLevels];
    int big[kBigCap];
    int bighit[kBigCap];
    int buf[NT / 32][64];
    unsigned long long walked_v, walked_e, scanned;
};

__device__ __forceinline__ bool bit_of(const uint32_t* B, int k) { return (B[k >> 5] >> (k & 31)) & 1u; }

__device__ __forceinline__ int nth_group(unsigned m, int g)
{
    for (int q = 0; q < g; ++q) m &= m - 1;  // drops the g lowest set bits
    return m ? __ffs(m) - 1 : -1;
}

// One vertex per lane (x where ok): act(v, k[4]) gets up to four neighbours k
// (-1 past the end) of a vertex whose value is v, from whichever lane scans
// them: short lists stay with their lane, up to kGroupDeg eight lanes share
// one, longer ones take the warp, and lists of kBigDeg and more are listed in
// sm.big for the whole CTA.  No block barrier inside.
template <int NT, class V, class Act>
__device__ __forceinline__ void push_batch(const DevGraph& G, StaticSmem<NT>& sm, int x, bool ok, V v, Act act)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int64_t rs = 0;
    int d = 0;
    if (ok) {
        rs = G.row[x];
        d = G.deg[x];
    }
    if (d >= kBigDeg) {
        const int p = atomicAdd(&sm.nbig, 1);
        if (p < kBigCap) {
            sm.big[p] = x;
            d = 0;
        }
    }
    if (d > 0 && d <= kThreadDeg) {
        int k[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) k[u] = u < d ? G.col[rs + u] : -1;
        act(v, k);
    }
    __syncwarp();
    for (unsigned m = __ballot_sync(full, d > kThreadDeg && d <= kGroupDeg); m;) {
        const int j = nth_group(m, lane >> 3);
        const int64_t rj = __shfl_sync(full, rs, j & 31);
        const int dj = __shfl_sync(full, d, j & 31);
        const V vj = __shfl_sync(full, v, j & 31);
        if (j >= 0)
            for (int s0 = lane & 7; s0 < dj; s0 += 32) {
                int k[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) k[u] = s0 + 8 * u < dj ? G.col[rj + s0 + 8 * u] : -1;
                act(vj, k);
            }
        __syncwarp();
        for (int q = 0; q < 4; ++q) m &= m - 1;
    }
    for (unsigned m = __ballot_sync(full, d > kGroupDeg); m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        const int64_t rj = __shfl_sync(full, rs, j);
        const int dj = __shfl_sync(full, d, j);
        const V vj = __shfl_sync(full, v, j);
        for (int s0 = lane; s0 < dj; s0 += 128) {
            int k[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) k[u] = s0 + 32 * u < dj ? G.col[rj + s0 + 32 * u] : -1;
            act(vj, k);
        }
        __syncwarp();
    }
}

// One vertex per lane: sums val(k) over the neighbours k with test(k), the
// lists shared out as in push_batch, and calls done(x, sum, whether any
// neighbour passed) in the lane that brought x.
template <int NT, class T, class Test, class Val, class Done>
__device__ __forceinline__ void pull_batch(const DevGraph& G, StaticSmem<NT>& sm, int x, bool ok, Test test, Val val,
                                           Done done)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int64_t rs = 0;
    int d = 0;
    if (ok) {
        rs = G.row[x];
        d = G.deg[x];
    }
    if (d >= kBigDeg) {
        const int p = atomicAdd(&sm.nbig, 1);
        if (p < kBigCap) {
            sm.big[p] = x;
            sm.bighit[p] = 0;
            d = 0;
            ok = false;  // finished by the whole CTA
        }
    }
    // four neighbours tested, then their values gathered, then summed
    auto four = [&](const int (&k)[4], T& s, bool& hit) {
        bool t[4];
        T y[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) t[u] = k[u] >= 0 && test(k[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) y[u] = t[u] ? val(k[u]) : (T)0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (t[u]) {
                s += y[u];
                hit = true;
            }
    };
    T sum = (T)0;
    bool hit = false;
    if (d > 0 && d <= kThreadDeg) {
        int k[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) k[u] = u < d ? G.col[rs + u] : -1;
        four(k, sum, hit);
    }
    __syncwarp();
    for (unsigned m = __ballot_sync(full, d > kThreadDeg && d <= kGroupDeg); m;) {
        const int j = nth_group(m, lane >> 3);
        const int64_t rj = __shfl_sync(full, rs, j & 31);
        const int dj = __shfl_sync(full, d, j & 31);
        T s = (T)0;
        bool h = false;
        if (j >= 0)
            for (int s0 = lane & 7; s0 < dj; s0 += 32) {
                int k[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) k[u] = s0 + 8 * u < dj ? G.col[rj + s0 + 8 * u] : -1;
                four(k, s, h);
            }
        const unsigned hits = __ballot_sync(full, h);
        if (hits) {
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(full, s, o);
        }
        // the vertex's own lane takes its group's total
        const int rank = __popc(m & ((1u << lane) - 1u));
        const T mine = __shfl_sync(full, s, (rank & 3) * 8);
        if (((m >> lane) & 1u) && rank < 4) {
            sum = mine;
            hit = (hits >> (rank * 8)) & 0xffu;
        }
        for (int q = 0; q < 4; ++q) m &= m - 1;
    }
    for (unsigned m = __ballot_sync(full, d > kGroupDeg); m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        const int64_t rj = __shfl_sync(full, rs, j);
        const int dj = __shfl_sync(full, d, j);
        T s = (T)0;
        bool h = false;
        for (int s0 = lane; s0 < dj; s0 += 128) {
            int k[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) k[u] = s0 + 32 * u < dj ? G.col[rj + s0 + 32 * u] : -1;
            four(k, s, h);
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
    if (ok) done(x, sum, hit);
    __syncwarp();
}

// Vertices of a list, handed to the warps in tasks of up to 32 (fewer when the
// list is short, so that every warp has work); batch(x, ok) per warp.
template <int NT, class Batch>
__device__ __forceinline__ void list_tasks(StaticSmem<NT>& sm, const int32_t* list, int n, Batch batch)
{
    const int lane = threadIdx.x & 31;
    const int t = min(32, max(1, (n + NT / 32 - 1) / (NT / 32)));
    for (;;) {
        int base = 0;
        if (lane == 0) base = atomicAdd(&sm.next, t);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n) break;
        const bool ok = lane < t && base + lane < n;
        batch(ok ? list[base + lane] : 0, ok);
    }
}

// The vertices whose bit in V is clear, packed 32 at a time per warp.
template <int NT, class Batch>
__device__ __forceinline__ void unset_tasks(StaticSmem<NT>& sm, const uint32_t* V, int nw, Batch batch)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int* buf = sm.buf[threadIdx.x >> 5];
    const int t = min(32, max(1, nw / (NT / 32)));
    int pend = 0;
    for (;;) {
        int base = 0;
        if (lane == 0) base = atomicAdd(&sm.next, t);
        base = __shfl_sync(full, base, 0);
        if (base >= nw) break;
        const unsigned mine = lane < t && base + lane < nw ? ~V[base + lane] : 0u;
        for (unsigned have = __ballot_sync(full, mine != 0u); have; have &= have - 1) {
            const int j = __ffs(have) - 1;
            const unsigned w = __shfl_sync(full, mine, j);
            if ((w >> lane) & 1u) buf[pend + __popc(w & ((1u << lane) - 1u))] = (base + j) * 32 + lane;
            pend += __popc(w);
            __syncwarp();
            if (pend >= 32) {
                batch(buf[lane], true);
                pend -= 32;
                const int rest = buf[32 + lane];
                __syncwarp();
                if (lane < pend) buf[lane] = rest;
                __syncwarp();
            }
        }
    }
    if (pend > 0) batch(lane < pend ? buf[lane] : 0, lane < pend);
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
//     backward, the parents pull or the children push.  On R-MAT graphs the
//     hubs sit on the middle levels, and 2.4 times fewer slots are scanned.
//   * Warps take vertices from the level by themselves (list_tasks): three
//     block barriers per level instead of five per 1,024 vertices, and the
//     counters come from the level sizes instead of shared atomics.
//   * Levels, histogram and rosters leave the kernel with the rows.
template <int NT, int MODE>
__global__ void __launch_bounds__(NT, 1024 / NT) k_static(const __grid_constant__ StaticArgs A)
{
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ StaticSmem<NT> sm;
    if (A.abort && *A.abort) return;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t nv = A.nv;
    const int nw = (int)((nv + 31) / 32);
    const bool sym = !A.asym && !(A.asym_dev && *A.asym_dev);

    // this worker's queue, level starts, child weights and bitmaps
    const size_t slot = blockIdx.x / A.halves;
    int32_t *qd, *lvl;
    double* acc;
    uint32_t *B, *V;  // tested bitmap, visited bitmap (isolated vertices count as visited)
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
    } else {
        const bool second = blockIdx.x % A.halves;
        qd = (second ? A.scr.qa : A.scr.qd) + slot * nv;
        lvl = second ? A.scr.qs + slot * nv : A.scr.lvl + slot * (size_t)(nv + 2);
        acc = (second ? (double*)A.scr.dp : A.scr.acc) + slot * nv;
        if (MODE == kBits) {
            V = (uint32_t*)s_dyn;
            B = V + nw;
        } else {
            V = A.scr.bits + slot * bitmap_words(nv);
            B = MODE == kOneBits ? (uint32_t*)s_dyn : (uint32_t*)(A.scr.st + slot * nv);
        }
    }
    if (threadIdx.x == 0) sm.walked_v = sm.walked_e = sm.scanned = 0;

    for (;;) {
        if (threadIdx.x == 0) {
            sm.item = atomicAdd(A.work_counter, 1);
            sm.total = 0;
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
            for (int64_t x = threadIdx.x; x < (int64_t)nw * 32; x += NT) {
                int d = 0;
                if (x < nv) {
                    d = A.G.deg[x];
                    D[x] = SBC_INF;
                    Sg[x] = 0;
                    if (MODE == kSmall) acc[x] = 0.0;
                }
                sum += (unsigned)d;
                const unsigned word = __ballot_sync(full, x >= nv || (sym && d == 0));
                if (lane == 0) V[x >> 5] = word;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(full, sum, o);
            if (lane == 0) atomicAdd(&sm.total, sum);
        }
        __syncthreads();
        const unsigned long long total = sm.total;
        int nlev = 0, reached = 0;
        unsigned long long visited = 0, scanned = 0;
        if (valid) {
            unsigned long long front = (unsigned)A.G.deg[root];
            if (threadIdx.x == 0) {
                D[root] = 0;
                Sg[root] = 1;
                qd[0] = root;
                lvl[0] = 0;
                sm.tail = 1;
                sm.lvslots[0] = front;
                V[root >> 5] |= 1u << (root & 31);
            }
            visited = front;
            // ---- forward: levels 0, 1, ... ----
            int L = 0, lo = 0, hi = 1;
            bool held = false;  // kOneBits: B is a copy of V
            for (;;) {
                const unsigned long long rest = total - visited;
                // the scan for unvisited vertices itself costs about a slot per four vertices
                const bool pull = sym && rest + (unsigned long long)(nv >> 2) < front;
                if (threadIdx.x == 0) sm.next = sm.nbig = 0;
                __syncthreads();
                if (threadIdx.x == 0) sm.slots = 0;
                if (!pull) {
                    scanned += front;
                    const uint32_t* T = V;
                    if (MODE == kOneBits) {
                        if (!held) {
                            for (int i = threadIdx.x; i < nw; i += NT) B[i] = V[i];
                            held = true;
                            __syncthreads();
                        }
                        T = B;
                    }
                    // an unvisited neighbour gains x's sigma; the first visitor
                    // (the one that finds sigma 0) claims it for the level.  A
                    // sum that wraps to 0 only makes more of them try.
                    auto act = [&](long long s, const int (&k)[4]) {
                        bool t[4];
                        unsigned long long old[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) t[u] = k[u] >= 0 && !bit_of(T, k[u]);
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            old[u] = t[u] ? atomicAdd((unsigned long long*)&Sg[k[u]], (unsigned long long)s) : 1ull;
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (old[u] == 0ull)
                                warp_append(&sm.tail, qd, k[u], atomicCAS(&D[k[u]], SBC_INF, L + 1) == SBC_INF);
                    };
                    list_tasks<NT>(sm, qd + lo, hi - lo, [&](int x, bool ok) {
                        push_batch<NT>(A.G, sm, x, ok, ok ? (long long)Sg[x] : 0ll, act);
                    });
                    __syncthreads();
                    for (int b = 0; b < min(sm.nbig, kBigCap); ++b) {
                        const int x = sm.big[b];
                        const int64_t rs = A.G.row[x];
                        const int d = A.G.deg[x];
                        const long long s = Sg[x];
                        for (int s0 = threadIdx.x; s0 < d; s0 += 4 * NT) {
                            int k[4];
#pragma unroll
                            for (int u = 0; u < 4; ++u) k[u] = s0 + NT * u < d ? A.G.col[rs + s0 + NT * u] : -1;
                            act(s, k);
                        }
                    }
                } else {
                    scanned += rest;
                    held = false;
                    for (int i = threadIdx.x; i < nw; i += NT) B[i] = 0u;
                    __syncthreads();
                    for (int i = lo + threadIdx.x; i < hi; i += NT) atomicOr(&B[qd[i] >> 5], 1u << (qd[i] & 31));
                    __syncthreads();
                    auto test = [&](int k) { return bit_of(B, k); };
                    auto val = [&](int k) { return (long long)Sg[k]; };
                    auto done = [&](int x, long long sum, bool hit) {
                        if (hit) {
                            D[x] = L + 1;
                            Sg[x] = sum;
                        }
                        warp_append(&sm.tail, qd, x, hit);
                    };
                    unset_tasks<NT>(sm, V, nw, [&](int x, bool ok) {
                        pull_batch<NT, long long>(A.G, sm, x, ok, test, val, done);
                    });
                    __syncthreads();
                    const int nb = min(sm.nbig, kBigCap);
                    for (int b = 0; b < nb; ++b) {
                        const int x = sm.big[b];
                        const int64_t rs = A.G.row[x];
                        const int d = A.G.deg[x];
                        long long s = 0;
                        bool h = false;
                        for (int s0 = threadIdx.x; s0 < d; s0 += NT) {
                            const int k = A.G.col[rs + s0];
                            if (test(k)) {
                                s += val(k);
                                h = true;
                            }
                        }
                        if (h) {
                            atomic_add_i64(&Sg[x], s);
                            sm.bighit[b] = 1;
                        }
                    }
                    if (nb > 0) {
                        __syncthreads();
                        for (int b = threadIdx.x; b < nb; b += NT)
                            done(sm.big[b], (long long)Sg[sm.big[b]], sm.bighit[b] != 0);
                    }
                }
                __syncthreads();
                lo = hi;
                hi = sm.tail;
                if (lo == hi) break;
                ++L;
                unsigned long long sum = 0;
                for (int i = lo + threadIdx.x; i < hi; i += NT) {
                    const int x = qd[i];
                    const unsigned bit = 1u << (x & 31);
                    atomicOr(&V[x >> 5], bit);
                    if (MODE == kOneBits && held) atomicOr(&B[x >> 5], bit);
                    sum += (unsigned)A.G.deg[x];
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(full, sum, o);
                if (lane == 0 && sum) atomicAdd(&sm.slots, sum);
                if (threadIdx.x == 0) lvl[L] = lo;
                __syncthreads();
                front = sm.slots;
                visited += front;
                if (threadIdx.x == 0 && L < kSlotLevels) sm.lvslots[L] = front;
            }
            nlev = L + 1;
            reached = hi;

            // ---- backward: each vertex sums its children's weights
            // w = (delta + 1) / sigma, kept in acc ----
            for (int i = threadIdx.x; i < nw; i += NT) B[i] = 0u;
            auto finish = [&](int x, double sum) {
                const double sx = (double)Sg[x];
                const double nd = sx * sum;
                Dl[x] = nd;
                acc[x] = (nd + 1.0) / sx;
            };
            for (int i = lvl[nlev - 1] + threadIdx.x; i < reached; i += NT) finish(qd[i], 0.0);
            __syncthreads();
            int end = reached;  // of level l + 1
            for (int l = nlev - 2; l >= 0; --l) {
                const int a0 = lvl[l], a1 = lvl[l + 1];
                const bool push = sym && l + 1 < kSlotLevels && sm.lvslots[l + 1] < sm.lvslots[l];
                const int m0 = push ? a0 : a1, m1 = push ? a1 : end;  // the level in the bitmap
                for (int i = m0 + threadIdx.x; i < m1; i += NT) atomicOr(&B[qd[i] >> 5], 1u << (qd[i] & 31));
                if (threadIdx.x == 0) {
                    sm.next = sm.nbig = 0;
                    if (l + 1 < kSlotLevels) sm.scanned += push ? sm.lvslots[l + 1] : sm.lvslots[l];
                }
                __syncthreads();
                if (push) {
                    auto act = [&](double w, const int (&k)[4]) {
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (k[u] >= 0 && bit_of(B, k[u])) atomicAdd(&acc[k[u]], w);
                    };
                    list_tasks<NT>(sm, qd + a1, end - a1, [&](int x, bool ok) {
                        push_batch<NT>(A.G, sm, x, ok, ok ? acc[x] : 0.0, act);
                    });
                    __syncthreads();
                    const int nb = min(sm.nbig, kBigCap);
                    for (int b = 0; b < nb; ++b) {
                        const int x = sm.big[b];
                        const int64_t rs = A.G.row[x];
                        const int d = A.G.deg[x];
                        const double w = acc[x];
                        for (int s0 = threadIdx.x; s0 < d; s0 += 4 * NT) {
                            int k[4];
#pragma unroll
                            for (int u = 0; u < 4; ++u) k[u] = s0 + NT * u < d ? A.G.col[rs + s0 + NT * u] : -1;
                            act(w, k);
                        }
                    }
                    if (nb > 0) __syncthreads();
                    for (int i = a0 + threadIdx.x; i < a1; i += NT) finish(qd[i], acc[qd[i]]);
                } else {
                    auto test = [&](int k) { return bit_of(B, k); };
                    auto val = [&](int k) { return acc[k]; };
                    list_tasks<NT>(sm, qd + a0, a1 - a0, [&](int x, bool ok) {
                        pull_batch<NT, double>(A.G, sm, x, ok, test, val,
                                               [&](int y, double sum, bool) { finish(y, sum); });
                    });
                    __syncthreads();
                    const int nb = min(sm.nbig, kBigCap);
                    for (int b = 0; b < nb; ++b) {
                        const int x = sm.big[b];
                        const int64_t rs = A.G.row[x];
                        const int d = A.G.deg[x];
                        double s = 0.0;
                        for (int s0 = threadIdx.x; s0 < d; s0 += NT) {
                            const int k = A.G.col[rs + s0];
                            if (test(k)) s += val(k);
                        }
                        if (__any_sync(full, s != 0.0)) {
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(full, s, o);
                            if (lane == 0) atomicAdd(&acc[x], s);
                        }
                    }
                    if (nb > 0) {
                        __syncthreads();
                        for (int b = threadIdx.x; b < nb; b += NT) finish(sm.big[b], acc[sm.big[b]]);
                    }
                }
                __syncthreads();
                for (int i = m0 + threadIdx.x; i < m1; i += NT) B[qd[i] >> 5] = 0u;
                __syncthreads();
                end = a1;
            }
        }

        // ---- the rows, and what is derived from the levels ----
        uint32_t* D2 = A.dist2 ? A.dist2 + (size_t)r * d2_words(nv) : nullptr;
        for (int64_t x = threadIdx.x; x < (int64_t)nw * 32; x += NT) {
            const int d = x < nv ? D[x] : SBC_INF;
            if (x < nv) {
                D8[x] = enc_d8(d);
                if (MODE == kSmall) {
                    gD[x] = d;
                    gS[x] = Sg[x];
                } else if (d != SBC_INF) {
                    acc[x] = 0.0;
                }
                if (d == SBC_INF) Dl[x] = 0.0;
            }
            if (D2) {
                // two bits per vertex: the ballots of the low and the high
                // bits, spread to even and odd places
                const unsigned c = enc_d2(d);
                unsigned even = __ballot_sync(full, c & 1u), odd = __ballot_sync(full, c & 2u);
                if (lane < 2) {
                    if (lane) {
                        even >>= 16;
                        odd >>= 16;
                    }
                    auto spread = [](unsigned v) {
                        v &= 0xffffu;
                        v = (v | (v << 8)) & 0x00ff00ffu;
                        v = (v | (v << 4)) & 0x0f0f0f0fu;
                        v = (v | (v << 2)) & 0x33333333u;
                        return (v | (v << 1)) & 0x55555555u;
                    };
                    const int64_t word = ((x - lane) >> 4) + lane;
                    if (word < d2_words(nv)) D2[word] = spread(even) | (spread(odd) << 1);
                }
            }
            if (MODE >= kOneBits && lane == 0) V[x >> 5] = 0u;
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
            sm.scanned += scanned;
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
// kSumCols vertices at a time and shares the roots out among kSumParts rows of
// threads (each in root order; the parts are added in order at the end): with a
// thread per vertex alone, a graph of 1,024 vertices summed its 1,024 roots on
// four blocks.
constexpr int kSumCols = 32, kSumParts = 16;

__global__ void __launch_bounds__(kSumCols* kSumParts) k_bc_colsum(const double* __restrict__ delta,
                                                                   const int64_t* __restrict__ roots, int nk,
                                                                   int64_t nv, double* __restrict__ bc,
                                                                   const int* __restrict__ abort)
{
    __shared__ double part[kSumParts][kSumCols];
    if (abort && *abort) return;
    const int c = threadIdx.x % kSumCols, p = threadIdx.x / kSumCols;
    const int per = (nk + kSumParts - 1) / kSumParts;
    const int r0 = min(nk, p * per), r1 = min(nk, r0 + per);
    for (int64_t v0 = blockIdx.x * (int64_t)kSumCols; v0 < nv; v0 += (int64_t)gridDim.x * kSumCols) {
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
            for (int q = 1; q < kSumParts; ++q) s += part[q][c];
            bc[v] = s;
        }
        __syncthreads();
    }
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

size_t static_dyn(int mode, int64_t nv)
{
    const size_t nw = (size_t)((nv + 31) / 32) * 4;
    return mode == kSmall ? (size_t)nv * 28 + 2 * nw : mode == kBits ? 2 * nw : mode == kOneBits ? nw : 0;
}

size_t static_fixed(int nt)
{
    return nt == 128 ? sizeof(StaticSmem<128>) : nt == 256 ? sizeof(StaticSmem<256>)
         : nt == 512 ? sizeof(StaticSmem<512>) : sizeof(StaticSmem<1024>);
}

StaticKernel static_kernel(int nt, int mode)
{
    if (mode == kSmall)
        return nt == 128 ? k_static<128, kSmall> : nt == 256 ? k_static<256, kSmall>
             : nt == 512 ? k_static<512, kSmall> : k_static<1024, kSmall>;
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
// worker's scratch has room for two static workers where both bitmaps are in
// shared memory.
StaticShape static_shape(int64_t nv, int64_t nk, int64_t workers, int sm_count, size_t smem_block, size_t smem_sm,
                         bool may_halve)
{
    StaticShape S;
    S.mode = kSmall;
    while (S.mode != kNoBits && static_dyn(S.mode, nv) + static_fixed(1024) + 1024 > smem_block) ++S.mode;
    S.dyn = static_dyn(S.mode, nv);
    S.halves = S.mode == kBits && may_halve ? 2 : 1;
    int64_t c = std::max<int64_t>(1, (nk + sm_count - 1) / sm_count);
    c = std::min<int64_t>(c, S.mode == kSmall ? 8 : S.mode == kBits ? 4 : 1);
    if (S.mode != kSmall) c = std::min<int64_t>(c, std::max<int64_t>(1, (workers * S.halves + sm_count - 1) / sm_count));
    // fewer CTAs while the SM's shared memory does not hold them (1 KB each is the system's)
    while (c > 1 && (size_t)c * (S.dyn + static_fixed(pow2_floor(1024 / c)) + 1024) > smem_sm) --c;
    S.nt = std::max(pow2_floor(1024 / c), S.mode == kSmall ? 128 : S.mode == kBits ? 256 : 1024);
    S.grid = (int)std::min<int64_t>(nk, c * sm_count);
    if (S.mode != kSmall) S.grid = (int)std::min<int64_t>(S.grid, workers * S.halves);
    S.kernel = static_kernel(S.nt, S.mode);
    return S;
}

cudaError_t static_launch(const StaticShape& S, const StaticArgs& A, cudaStream_t s)
{
    if (S.dyn + static_fixed(S.nt) > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(S.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S.dyn);
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
    f->prof_begin(PROF_STATIC);
    e = static_launch(S, A, s);
    f->prof_end(PROF_STATIC);
    if (e) return e;
    if (d_list) return cudaSuccess;  // the caller moves BC by the listed roots' old and new rows
    const int bgrid = (int)std::min<int64_t>((f->nv + kSumCols - 1) / kSumCols, (int64_t)f->sm_count * 64);
    k_bc_colsum<<<std::max(bgrid, 1), kSumCols * kSumParts, 0, s>>>(f->d_delta, f->d_roots, (int)f->nk, f->nv,
                                                                    f->d_bc, nullptr);
    return cudaGetLastError();
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
// neighbour ids).  k_static and k_bc_colsum_checked read the word and do
// nothing when it is set, so a bad id never becomes an out-of-bounds access.
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
    if (static_launch(S, A, s) != cudaSuccess) return noalloc_fail(SBC_ERR_CUDA, "sbc_static_init_noalloc: k_static launch failed");
    const int bgrid = (int)std::min<int64_t>((nv + kSumCols - 1) / kSumCols, 8192);
    k_bc_colsum<<<bgrid, kSumCols * kSumParts, 0, s>>>(d_delta, d_roots, (int)nk, nv, d_bc, bad);
    if (noalloc_launch_failed("k_bc_colsum", &rc)) return rc;
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
