// Device slack-CSR adjacency: in-place insertion and re-pack.
//
// Replaces stinger_insert_edge (src/stinger/stinger.c:778-876) and the edge
// block pool.  Each vertex owns slots [row[v], row[v]+cap[v]); the first deg[v]
// hold live neighbours.  An insertion appends into the slack of both endpoints
// (one direction for the directed form) after a duplicate check, and stamps the
// slot with the insertion's index inside its batch (seq), so that a traversal
// for insertion i of a batch sees only edges of insertions <= i.
#include <climits>
#include "sbc_host.h"
#include "sbc_internal.cuh"

namespace sbc {

// Insertion outcome codes written to ok[i]:
//   1 inserted, 0 duplicate (edge already present), -1 self loop or id out of
//   range, -2 no slack left (the host plans capacity so this is not expected).
__device__ __forceinline__ void append_warp(int64_t nv, const int64_t* __restrict__ row, int32_t* deg,
                                            const int32_t* __restrict__ cap, int32_t* col, int32_t* seq, int n,
                                            const int32_t* __restrict__ iu, const int32_t* __restrict__ iv,
                                            int32_t* ok, int directed, int* err)
{
    const int lane = threadIdx.x;
    for (int i = 0; i < n; ++i) {
        const int u = iu[i], v = iv[i];
        int code = 1;
        if (u == v || u < 0 || v < 0 || u >= nv || v >= nv) code = -1;
        if (code == 1) {
            int x = u, y = v;
            if (!directed && deg[v] < deg[u]) {
                x = v;
                y = u;
            }
            const int dx = deg[x];
            const int64_t rx = row[x];
            bool found = false;
            for (int s = lane; s < dx; s += 32)
                if (col[rx + s] == y) found = true;
            if (__any_sync(0xffffffffu, found)) code = 0;
        }
        if (code == 1 && !(deg[u] < cap[u] && (directed || deg[v] < cap[v]))) {
            code = -2;
            if (lane == 0) atomicOr(err, 1);
        }
        if (lane == 0) {
            if (code == 1) {
                int p = deg[u];
                col[row[u] + p] = v;
                seq[row[u] + p] = i;
                deg[u] = p + 1;
                if (!directed) {
                    p = deg[v];
                    col[row[v] + p] = u;
                    seq[row[v] + p] = i;
                    deg[v] = p + 1;
                }
            }
            ok[i] = code;
        }
        __syncwarp();
    }
}

__global__ void k_append(int64_t nv, const int64_t* __restrict__ row, int32_t* deg, const int32_t* __restrict__ cap,
                         int32_t* col, int32_t* seq, int n, const int32_t* __restrict__ iu,
                         const int32_t* __restrict__ iv, int32_t* ok, int directed, int* err)
{
    append_warp(nv, row, deg, cap, col, seq, n, iu, iv, ok, directed, err);
}

// First slot of x in [0, ns) whose neighbour is >= y, 32 probes a step.
__device__ __forceinline__ int warp_lower_bound(const int32_t* __restrict__ col, int64_t rx, int ns, int y)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = ns;
    while (hi > lo) {
        const int step = (hi - lo + 31) >> 5;
        const int64_t p = lo + (int64_t)lane * step;
        const int below = __popc(__ballot_sync(full, p < hi && col[rx + p] < y));  // probes ascend: the first `below`
        const int base = lo;
        if (below == 0) return base;
        lo = (int)min((int64_t)hi, base + (int64_t)(below - 1) * step + 1);
        hi = (int)min((int64_t)hi, base + (int64_t)below * step);
    }
    return lo;
}

// Whether y is among x's d slots, the first ns of which are sorted (one warp).
__device__ __forceinline__ bool has_slot(const int32_t* col, int64_t rx, int ns, int d, int y)
{
    const int lane = threadIdx.x & 31;
    const int p = warp_lower_bound(col, rx, ns, y);
    bool found = p < ns && col[rx + p] == y;
    for (int s = ns + lane; s < d; s += 32)
        if (col[rx + s] == y) found = true;
    return __any_sync(0xffffffffu, found);
}

// The same results with a warp per insertion, in three launches:
//   k_append_codes  -1 bad id or loop; 0 an edge already (of the graph as the
//                   batch begins -- sealed, so a binary search of the sorted
//                   slots plus a scan of any tail -- or of an earlier
//                   insertion of the batch); 1 to insert.
//   k_append_rank   each insertion's rank among the batch's insertions at
//                   each endpoint (its slot past deg0, so that every vertex's
//                   appended slots stay in insertion order), and whether
//                   every slot fits the vertex's slack.
//   k_append_place  the slots written (seq = index) and the degrees raised;
//                   if some slot does not fit, one warp appends the whole
//                   batch in order instead (k_append's way), so that exactly
//                   the insertions a one-by-one append rejects are rejected.
// rk holds 2 n ranks and, at rk[2 n], the misfit flag.
__global__ void k_append_codes(int64_t nv, const int64_t* __restrict__ row, const int32_t* __restrict__ deg,
                               const int32_t* __restrict__ nsort, const int32_t* __restrict__ col, int n,
                               const int32_t* __restrict__ iu, const int32_t* __restrict__ iv, int32_t* ok,
                               int directed, int32_t* rk)
{
    const int w = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (w == 0 && lane == 0) rk[2 * n] = 0;
    if (w >= n) return;
    const int u = iu[w], v = iv[w];
    int code = (u == v || u < 0 || v < 0 || u >= nv || v >= nv) ? -1 : 1;
    if (code == 1) {
        bool dup = false;
        for (int base = 0; base < w && !dup; base += 32) {
            const int j = base + lane;
            bool same = false;
            if (j < w) {
                const int a = iu[j], b = iv[j];
                same = (a == u && b == v) || (!directed && a == v && b == u);
            }
            dup = __any_sync(0xffffffffu, same);
        }
        if (dup) code = 0;
    }
    if (code == 1) {
        int x = u, y = v;
        if (!directed && deg[v] < deg[u]) {
            x = v;
            y = u;
        }
        const int64_t rx = row[x];
        const int d = deg[x], ns = min(nsort[x], d);
        if (has_slot(col, rx, ns, d, y)) code = 0;
    }
    if (lane == 0) ok[w] = code;
}

__global__ void k_append_rank(const int32_t* __restrict__ deg0, const int32_t* __restrict__ cap, int n,
                              const int32_t* __restrict__ iu, const int32_t* __restrict__ iv,
                              const int32_t* __restrict__ ok, int directed, int32_t* rk)
{
    const int w = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (w >= n || ok[w] != 1) return;
    const int u = iu[w], v = iv[w];
    int ru = 0, rv = 0;
    for (int j = lane; j < w; j += 32) {
        if (ok[j] != 1) continue;
        const int a = iu[j], b = iv[j];
        ru += (a == u || (!directed && b == u)) ? 1 : 0;
        rv += (a == v || b == v) ? 1 : 0;
    }
    ru = __reduce_add_sync(0xffffffffu, ru);
    rv = __reduce_add_sync(0xffffffffu, rv);
    if (lane == 0) {
        rk[w] = ru;
        rk[n + w] = rv;
        if (deg0[u] + ru >= cap[u] || (!directed && deg0[v] + rv >= cap[v])) atomicOr(&rk[2 * n], 1);
    }
}

__global__ void k_append_place(int64_t nv, const int64_t* __restrict__ row, int32_t* deg,
                               const int32_t* __restrict__ deg0, const int32_t* __restrict__ cap, int32_t* col,
                               int32_t* seq, int n, const int32_t* __restrict__ iu, const int32_t* __restrict__ iv,
                               int32_t* ok, int directed, const int32_t* __restrict__ rk, int* err)
{
    if (rk[2 * n]) {
        // a slot does not fit: the whole batch in order, one warp
        if (blockIdx.x == 0 && threadIdx.x < 32)
            append_warp(nv, row, deg, cap, col, seq, n, iu, iv, ok, directed, err);
        return;
    }
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || ok[i] != 1) return;
    const int u = iu[i], v = iv[i];
    const int pu = deg0[u] + rk[i];
    col[row[u] + pu] = v;
    seq[row[u] + pu] = i;
    atomicMax(&deg[u], pu + 1);
    if (!directed) {
        const int pv = deg0[v] + rk[n + i];
        col[row[v] + pv] = u;
        seq[row[v] + pv] = i;
        atomicMax(&deg[v], pv + 1);
    }
}

// The three steps in one CTA, a warp per insertion at a time: the batch and its
// codes are held in shared memory and barriers stand where the launches were.
// The time is that of a few dependent loads per round of warps, so a short
// batch costs one launch instead of three and a graph of a group does not take
// its insertions one after the other.  With the seal done by the merge: a step
// of one insertion and one deletion on ER 200 360 -> 347 us; 16 R-MAT graphs,
// 16 insertions each, where one warp per graph appended for 51 us: 10.28 ->
// 10.20 ms.  At two rounds of the CTA's 32 warps it measures the same as the
// three launches (a step of 37 on R-MAT 17 4.67 and 4.66 ms, of 64 on Chung-Lu
// 40k 4.15 both ways); beyond that a graph's batch keeps the launches.
constexpr int kBlockAppendMax = 256;  // insertions per CTA
constexpr int kFusedAppendMax = 64;   // one graph's batch

__device__ __forceinline__ void append_block(int64_t nv, const int64_t* row, int32_t* deg, const int32_t* deg0,
                                             const int32_t* nsort, const int32_t* cap, int32_t* col, int32_t* seq,
                                             int n, const int32_t* iu, const int32_t* iv, int32_t* ok, int directed,
                                             int* err)
{
    __shared__ int s_u[kBlockAppendMax], s_v[kBlockAppendMax], s_ok[kBlockAppendMax];
    __shared__ int s_ru[kBlockAppendMax], s_rv[kBlockAppendMax];
    __shared__ int s_misfit;
    const int lane = threadIdx.x & 31, warps = (int)(blockDim.x >> 5);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        s_u[i] = iu[i];
        s_v[i] = iv[i];
    }
    if (threadIdx.x == 0) s_misfit = 0;
    __syncthreads();
    for (int w = (int)(threadIdx.x >> 5); w < n; w += warps) {
        const int u = s_u[w], v = s_v[w];
        int code = (u == v || u < 0 || v < 0 || u >= nv || v >= nv) ? -1 : 1;
        if (code == 1) {
            bool same = false;
            for (int j = lane; j < w; j += 32)
                same |= (s_u[j] == u && s_v[j] == v) || (!directed && s_u[j] == v && s_v[j] == u);
            if (__any_sync(0xffffffffu, same)) code = 0;
        }
        if (code == 1) {
            const bool swap = !directed && deg[v] < deg[u];
            const int x = swap ? v : u;
            const int d = deg[x];
            if (has_slot(col, row[x], min(nsort[x], d), d, swap ? u : v)) code = 0;
        }
        if (lane == 0) s_ok[w] = code;
    }
    __syncthreads();
    for (int w = (int)(threadIdx.x >> 5); w < n; w += warps) {
        if (s_ok[w] != 1) continue;
        const int u = s_u[w], v = s_v[w];
        int ru = 0, rv = 0;
        for (int j = lane; j < w; j += 32) {
            if (s_ok[j] != 1) continue;
            ru += (s_u[j] == u || (!directed && s_v[j] == u)) ? 1 : 0;
            rv += ((!directed && s_u[j] == v) || s_v[j] == v) ? 1 : 0;
        }
        ru = __reduce_add_sync(0xffffffffu, ru);
        rv = __reduce_add_sync(0xffffffffu, rv);
        if (lane == 0) {
            s_ru[w] = ru;
            s_rv[w] = rv;
            if (deg0[u] + ru >= cap[u] || (!directed && deg0[v] + rv >= cap[v])) s_misfit = 1;
        }
    }
    __syncthreads();
    if (s_misfit) {
        // a slot does not fit: the whole batch in order, one warp
        if (threadIdx.x < 32) append_warp(nv, row, deg, cap, col, seq, n, iu, iv, ok, directed, err);
        return;
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        ok[i] = s_ok[i];
        if (s_ok[i] != 1) continue;
        const int u = s_u[i], v = s_v[i];
        const int pu = deg0[u] + s_ru[i];
        col[row[u] + pu] = v;
        seq[row[u] + pu] = i;
        atomicMax(&deg[u], pu + 1);
        if (!directed) {
            const int pv = deg0[v] + s_rv[i];
            col[row[v] + pv] = u;
            seq[row[v] + pv] = i;
            atomicMax(&deg[v], pv + 1);
        }
    }
}

__global__ void __launch_bounds__(1024) k_append_small(int64_t nv, const int64_t* row, int32_t* deg,
                                                       const int32_t* deg0, const int32_t* nsort, const int32_t* cap,
                                                       int32_t* col, int32_t* seq, int n, const int32_t* iu,
                                                       const int32_t* iv, int32_t* ok, int directed, int* err)
{
    append_block(nv, row, deg, deg0, nsort, cap, col, seq, n, iu, iv, ok, directed, err);
}

// Many graphs' batches at once, a CTA per graph; a batch too long for the
// CTA's tables is appended in order by one warp.
__global__ void __launch_bounds__(1024) k_append_group(const __grid_constant__ GraphBatchSlots S)
{
    const GraphBatchSlot& b = S.slot[blockIdx.x];
    if (b.n <= kBlockAppendMax)
        append_block(b.nv, b.row, b.deg, b.deg0, b.nsort, b.cap, b.col, b.seq, b.n, b.iu, b.iv, b.ok, 0, b.err);
    else if (threadIdx.x < 32)
        append_warp(b.nv, b.row, b.deg, b.cap, b.col, b.seq, b.n, b.iu, b.iv, b.ok, 0, b.err);
}

// A batch's endpoint arrays live in the caller's device memory.  k_set_src
// records their addresses in the graph's two-pointer slot (its arguments are
// copied at launch, so nothing on the host has to outlive the call), and
// k_stage_inputs, which a captured batch graph replays unchanged, copies from
// the addresses in the slot into the staging rows (u at dst[0..n), v at
// dst[cap..cap+n)).
__global__ void k_set_src(const int32_t** slot, const int32_t* u, const int32_t* v)
{
    slot[0] = u;
    slot[1] = v;
}

__global__ void k_stage_inputs(const int32_t* const* __restrict__ slot, int32_t* dst, int cap, int n)
{
    const int32_t* u = slot[0];
    const int32_t* v = slot[1];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        dst[i] = u[i];
        dst[cap + i] = v[i];
    }
}

cudaError_t launch_set_src(sbc_graph* g, const int32_t* d_u, const int32_t* d_v)
{
    k_set_src<<<1, 1, 0, g->stream>>>(g->d_src, d_u, d_v);
    return cudaGetLastError();
}

cudaError_t launch_stage(sbc_graph* g, int n)
{
    const int blocks = std::min((n + 255) / 256, 1024);
    k_stage_inputs<<<blocks < 1 ? 1 : blocks, 256, 0, g->stream>>>(g->d_src, g->d_ins, g->ins_capacity, n);
    return cudaGetLastError();
}

// After a batch's update: the slots it appended to a vertex (an unsorted tail
// after the first nsort[x] slots, which are sorted by neighbour id) are merged
// into the sorted prefix, so that edge tests (has_edge: binary search of the
// prefix, then a scan of the tail) never scan more than the current batch's
// appends -- without this a hub's tail grew by every insertion on it.  One
// block per endpoint of an applied insertion; the first block to reach a
// vertex claims it by swapping its deg0 for -1 and, when it is done, seals it:
// deg0 = deg makes the appended slots visible to all later traversals (the
// update that read deg0 has finished).  A block that finds deg0 = deg comes
// after the claimer (an appended slot leaves deg0 < deg) and puts it back.
// The tail (at most kMergeTail slots per batch; a longer one is merged over
// several batches) is sorted in shared memory; each tail value's final slot is
// its rank among the tail plus its lower bound in the prefix; prefix values
// move up by the number of tail values below them, in chunks from the end, so
// no value is overwritten before it is read.  seq of the moved slots is not
// read again (after the seal every slot is below deg0).
constexpr int kMergeTail = 2048;
constexpr int kMergeThreads = 256;
constexpr int kMergeRun = 8;  // prefix values per thread per chunk

__device__ __forceinline__ void merge_tail(const int64_t* __restrict__ row, const int32_t* __restrict__ deg,
                                           int32_t* deg0, int32_t* nsort, int32_t* col, int x)
{
    __shared__ int s_tail[kMergeTail];
    __shared__ int s_dst[kMergeTail];
    __shared__ int s_claim;
    const int tid = threadIdx.x;
    const int dx = deg[x];
    if (tid == 0) s_claim = atomicExch(&deg0[x], -1);
    __syncthreads();
    if (s_claim < 0) return;  // another block merges x
    const int ns = nsort[x];
    const int t = s_claim == dx ? 0 : min(dx - ns, kMergeTail);
    if (t <= 0) {  // no appended slots, or another block has merged them and left
        if (tid == 0) deg0[x] = dx;
        return;
    }
    const int64_t rx = row[x];
    int P = 1;
    while (P < t) P <<= 1;
    for (int k = tid; k < P; k += kMergeThreads) s_tail[k] = k < t ? col[rx + ns + k] : INT_MAX;
    __syncthreads();
    for (int size = 2; size <= P; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = tid; i < (P >> 1); i += kMergeThreads) {
                const int lo = (i / stride) * 2 * stride + (i % stride);
                const int hi = lo + stride;
                const int a = s_tail[lo], b = s_tail[hi];
                if ((a > b) == ((lo & size) == 0)) {
                    s_tail[lo] = b;
                    s_tail[hi] = a;
                }
            }
            __syncthreads();
        }
    }
    for (int k = tid; k < t; k += kMergeThreads) {
        const int v = s_tail[k];
        int lo = 0, hi = ns;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (col[rx + mid] < v) lo = mid + 1;
            else hi = mid;
        }
        s_dst[k] = lo + k;
    }
    __syncthreads();
    const int first = s_dst[0];  // prefix values below it stay where they are
    constexpr int kChunk = kMergeThreads * kMergeRun;
    for (int c1 = ns; c1 > first; c1 -= kChunk) {
        const int c0 = max(first, c1 - kChunk);
        int val[kMergeRun], dst[kMergeRun];
#pragma unroll
        for (int r = 0; r < kMergeRun; ++r) {
            const int idx = c0 + tid + r * kMergeThreads;
            dst[r] = -1;
            if (idx < c1) {
                const int v = col[rx + idx];
                int lo = 0, hi = t;  // tail values below v
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (s_tail[mid] < v) lo = mid + 1;
                    else hi = mid;
                }
                val[r] = v;
                dst[r] = idx + lo;
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kMergeRun; ++r)
            if (dst[r] >= 0) col[rx + dst[r]] = val[r];
        __syncthreads();
    }
    for (int k = tid; k < t; k += kMergeThreads) col[rx + s_dst[k]] = s_tail[k];
    if (tid == 0) {
        nsort[x] = ns + t;
        deg0[x] = dx;
    }
}

__global__ void __launch_bounds__(kMergeThreads) k_merge_tails(int n, const int32_t* __restrict__ iu,
                                                               const int32_t* __restrict__ iv,
                                                               const int32_t* __restrict__ ok,
                                                               const int64_t* __restrict__ row,
                                                               const int32_t* __restrict__ deg, int32_t* deg0,
                                                               int32_t* nsort, int32_t* col)
{
    const int e = blockIdx.x;
    const int i = e < n ? e : e - n;
    if (ok[i] <= 0) return;
    merge_tail(row, deg, deg0, nsort, col, e < n ? iu[i] : iv[i]);
}

// k_merge_tails over many graphs: blockIdx.y selects the graph.
__global__ void __launch_bounds__(kMergeThreads) k_merge_tails_group(const __grid_constant__ GraphBatchSlots S)
{
    const GraphBatchSlot& b = S.slot[blockIdx.y];
    const int e = blockIdx.x;
    if (S.errs && e == 0 && threadIdx.x == 0) S.errs[blockIdx.y] = *b.err;
    if (e >= 2 * b.n) return;
    const int i = e < b.n ? e : e - b.n;
    if (b.ok[i] <= 0) return;
    merge_tail(b.row, b.deg, b.deg0, b.nsort, b.col, e < b.n ? b.iu[i] : b.iv[i]);
}

// Removes neighbour y from x's slots (one warp): the slot is found, the later
// slots move down one place (a sorted prefix stays sorted), and deg -- and
// deg0 / nsort when the slot lay below them -- drop by one.  Returns whether y
// was present.
__device__ __forceinline__ bool remove_slot(const int64_t* __restrict__ row, int32_t* deg, int32_t* deg0,
                                            int32_t* nsort, int32_t* col, int32_t* seq, int x, int y)
{
    const int lane = threadIdx.x & 31;
    const int d = deg[x];
    const int64_t rx = row[x];
    int p = -1;
    for (int base = 0; base < d && p < 0; base += 32) {
        const int s = base + lane;
        const unsigned m = __ballot_sync(0xffffffffu, s < d && col[rx + s] == y);
        if (m) p = base + __ffs(m) - 1;
    }
    if (p < 0) return false;
    for (int base = p; base < d - 1; base += 32) {
        const int s = base + lane;
        int c = 0, q = 0;
        if (s < d - 1) {
            c = col[rx + s + 1];
            q = seq[rx + s + 1];
        }
        __syncwarp();  // every lane has read before any slot is overwritten
        if (s < d - 1) {
            col[rx + s] = c;
            seq[rx + s] = q;
        }
        __syncwarp();
    }
    if (lane == 0) {
        deg[x] = d - 1;
        if (p < deg0[x]) deg0[x] -= 1;
        if (p < nsort[x]) nsort[x] -= 1;
    }
    __syncwarp();
    return true;
}

// Edge removal (stinger_remove_edge, src/stinger/stinger.c): (u,v) and,
// unless directed, (v,u); *res = 1 removed, 0 absent, -1 self loop or id out
// of range.  One warp; the graph's stream orders it with the batches.
__global__ void k_remove(int64_t nv, const int64_t* __restrict__ row, int32_t* deg, int32_t* deg0, int32_t* nsort,
                         int32_t* col, int32_t* seq, int u, int v, int directed, int* res)
{
    int code;
    if (u == v || u < 0 || v < 0 || u >= nv || v >= nv) {
        code = -1;
    } else {
        code = remove_slot(row, deg, deg0, nsort, col, seq, u, v) ? 1 : 0;
        if (!directed) remove_slot(row, deg, deg0, nsort, col, seq, v, u);
    }
    if (threadIdx.x == 0) *res = code;
}

// Batched deletions, step 1: the n staged edges (iu/iv, -1 = invalid id) are
// removed in order, each only marked -- its two slots keep their place and get
// seq = -1 - i -- so that every deletion's update can still see the graph as
// it stood before it (a slot removed at deletion j is an edge for jobs i < j).
// code[i] = 1 removed, 0 absent (never there, or removed earlier in the
// batch), -1 self loop / bad id.
//
// Warp per deletion.  Every slot is live as the call begins, so what deletion
// i finds depends on earlier ones only through the number `nth` of them that
// name the same edge: a slot among the sorted leading ones is taken by the
// first of them, and in an unsorted tail (lists longer than one batch's merge)
// the nth match is.  By one thread in order, each of its two binary searches a
// chain of dependent loads, a batch of 256 on R-MAT 20 took 1.7 ms.

// The slot of x that the deletion with `nth` earlier ones of its edge removes, or -1.
__device__ __forceinline__ int64_t nth_slot(const int64_t* __restrict__ row, const int32_t* __restrict__ deg,
                                            const int32_t* __restrict__ nsort, const int32_t* __restrict__ col, int x,
                                            int y, int nth)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t rx = row[x];
    const int d = deg[x], ns = min(nsort[x], d);
    const int p = warp_lower_bound(col, rx, ns, y);
    if (p < ns && col[rx + p] == y) return nth == 0 ? rx + p : -1;
    for (int base = ns; base < d; base += 32) {
        const int s = base + lane;
        unsigned m = __ballot_sync(full, s < d && col[rx + s] == y);
        const int c = __popc(m);
        if (nth < c) {
            for (; nth > 0; --nth) m &= m - 1;
            return rx + base + __ffs(m) - 1;
        }
        nth -= c;
    }
    return -1;
}

__global__ void k_mark_removed(const int64_t* __restrict__ row, const int32_t* __restrict__ deg,
                               const int32_t* __restrict__ nsort, const int32_t* __restrict__ col, int32_t* seq, int n,
                               const int32_t* __restrict__ iu, const int32_t* __restrict__ iv, int32_t* code)
{
    const int i = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= n) return;
    const int u = iu[i], v = iv[i];
    if (u < 0 || v < 0 || u == v) {
        if (lane == 0) code[i] = -1;
        return;
    }
    int nth = 0;
    for (int j = lane; j < i; j += 32) {
        const int a = iu[j], b = iv[j];
        nth += ((a == u && b == v) || (a == v && b == u)) ? 1 : 0;
    }
    nth = __reduce_add_sync(0xffffffffu, nth);
    const int64_t pu = nth_slot(row, deg, nsort, col, u, v, nth);
    const int64_t pv = pu < 0 ? -1 : nth_slot(row, deg, nsort, col, v, u, nth);
    if (lane == 0) {
        code[i] = pv >= 0 ? 1 : 0;
        if (pv >= 0) {
            seq[pu] = -1 - i;
            seq[pv] = -1 - i;
        }
    }
}

// Batched deletions, step 3 (after the update): the marked slots leave their
// lists, which keep their order.  CTA per deletion endpoint; the first CTA to
// reach a vertex claims it by swapping its deg0 (== deg between batches) for
// -1, and CTAs that find it claimed leave it.  The claim outlives the launch
// (k_reopen ends it): a CTA that came after a claim was given up would read
// the vertex's degree and slots as its own SM last cached them, and put slots
// back that had left the list.  A single deletion has two endpoints and no
// second comer, so its CTAs end their claims themselves.
__global__ void __launch_bounds__(256) k_compact_removed(const int64_t* __restrict__ row, int32_t* deg, int32_t* deg0,
                                                         int32_t* nsort, int32_t* col, int32_t* seq, int n,
                                                         const int32_t* __restrict__ iu,
                                                         const int32_t* __restrict__ iv,
                                                         const int32_t* __restrict__ code)
{
    __shared__ int s_warp[8];
    __shared__ int s_keep_sorted;
    __shared__ int s_mine;
    const int i = blockIdx.x >> 1;
    if (code[i] != 1) return;
    const int x = (blockIdx.x & 1) ? iv[i] : iu[i];
    if (threadIdx.x == 0) s_mine = atomicExch(&deg0[x], -1) >= 0;
    __syncthreads();
    if (!s_mine) return;
    const int64_t rx = row[x];
    const int d = deg[x], ns = min(nsort[x], d);
    if (threadIdx.x == 0) s_keep_sorted = 0;
    int kept = 0;
    for (int base = 0; base < d; base += 256) {
        const int sl = base + (int)threadIdx.x;
        int c = 0, q = 0;
        bool keep = false;
        if (sl < d) {
            c = col[rx + sl];
            q = seq[rx + sl];
            keep = q >= 0;
        }
        int total;
        const int off = block_exclusive_scan<256>(keep ? 1 : 0, s_warp, &total);  // every read precedes its barrier
        if (keep) {
            col[rx + kept + off] = c;
            seq[rx + kept + off] = q;
        }
        if (keep && sl < ns) atomicAdd(&s_keep_sorted, 1);
        kept += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        deg[x] = kept;
        if (n == 1) deg0[x] = kept;
        nsort[x] = s_keep_sorted;
    }
}

// Ends the claims of k_compact_removed.
__global__ void k_reopen(const int32_t* __restrict__ deg, int32_t* deg0, int n, const int32_t* __restrict__ iu,
                         const int32_t* __restrict__ iv, const int32_t* __restrict__ code)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || code[i] != 1) return;
    deg0[iu[i]] = deg[iu[i]];
    deg0[iv[i]] = deg[iv[i]];
}

// Copy every vertex's live slots to a new layout with larger slack (warp per vertex).
__global__ void k_repack(int64_t nv, const int64_t* __restrict__ orow, const int32_t* __restrict__ deg,
                         const int32_t* __restrict__ ocol, const int32_t* __restrict__ oseq,
                         const int64_t* __restrict__ nrow, int32_t* __restrict__ ncol, int32_t* __restrict__ nseq)
{
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < nv; v += nwarps) {
        const int d = deg[v];
        const int64_t a = orow[v], b = nrow[v];
        for (int s = lane; s < d; s += 32) {
            ncol[b + s] = ocol[a + s];
            nseq[b + s] = oseq[a + s];
        }
    }
}

cudaError_t launch_append(sbc_graph* g, int n, bool directed)
{
    const int32_t* iu = g->d_ins;
    const int32_t* iv = g->d_ins + g->ins_capacity;
    int32_t* ok = g->d_ins + 2 * g->ins_capacity;
    g->last_directed = directed;
    if (n <= 0) return cudaSuccess;
    if (n > kParallelAppendMax) {
        // the parallel form's within-batch tests grow with n^2
        k_append<<<1, 32, 0, g->stream>>>(g->nv, g->d_row, g->d_deg, g->d_cap, g->d_col, g->d_seq, n, iu, iv, ok,
                                          directed ? 1 : 0, g->d_err);
        return cudaGetLastError();
    }
    if (n <= kFusedAppendMax) {
        k_append_small<<<1, 32 * std::min(n, 32), 0, g->stream>>>(g->nv, g->d_row, g->d_deg, g->d_deg0, g->d_nsort,
                                                                  g->d_cap, g->d_col, g->d_seq, n, iu, iv, ok,
                                                                  directed ? 1 : 0, g->d_err);
        return cudaGetLastError();
    }
    int32_t* rk = g->d_ins + 3 * g->ins_capacity;
    const int wblocks = (n + 7) / 8;  // 8 warps of 32 per block, a warp per insertion
    k_append_codes<<<wblocks, 256, 0, g->stream>>>(g->nv, g->d_row, g->d_deg, g->d_nsort, g->d_col, n, iu, iv, ok,
                                                   directed ? 1 : 0, rk);
    k_append_rank<<<wblocks, 256, 0, g->stream>>>(g->d_deg0, g->d_cap, n, iu, iv, ok, directed ? 1 : 0, rk);
    k_append_place<<<(n + 255) / 256, 256, 0, g->stream>>>(g->nv, g->d_row, g->d_deg, g->d_deg0, g->d_cap, g->d_col,
                                                           g->d_seq, n, iu, iv, ok, directed ? 1 : 0, rk, g->d_err);
    return cudaGetLastError();
}

cudaError_t launch_seal(sbc_graph* g, int n)
{
    const int32_t* iu = g->d_ins;
    const int32_t* iv = g->d_ins + g->ins_capacity;
    const int32_t* ok = g->d_ins + 2 * g->ins_capacity;
    if (n <= 0) return cudaSuccess;
    k_merge_tails<<<2 * n, kMergeThreads, 0, g->stream>>>(n, iu, iv, ok, g->d_row, g->d_deg, g->d_deg0, g->d_nsort,
                                                          g->d_col);
    cudaError_t e = cudaGetLastError();
    if (e) return e;
    return launch_l2mask_insert(g, n, g->last_directed);
}

GraphBatchSlot graph_batch_slot(sbc_graph* g, int n)
{
    GraphBatchSlot b;
    b.nv = g->nv;
    b.row = g->d_row;
    b.deg = g->d_deg;
    b.deg0 = g->d_deg0;
    b.nsort = g->d_nsort;
    b.cap = g->d_cap;
    b.col = g->d_col;
    b.seq = g->d_seq;
    b.iu = g->d_ins;
    b.iv = g->d_ins + g->ins_capacity;
    b.ok = g->d_ins + 2 * g->ins_capacity;
    b.err = g->d_err;
    b.n = n;
    return b;
}

cudaError_t launch_append_group(const GraphBatchSlots& S, cudaStream_t s)
{
    if (S.count <= 0) return cudaSuccess;
    int nmax = 0;
    for (int i = 0; i < S.count; ++i) nmax = std::max(nmax, S.slot[i].n);
    k_append_group<<<S.count, 32 * std::min(std::max(nmax, 1), 32), 0, s>>>(S);
    return cudaGetLastError();
}

cudaError_t launch_seal_group(const GraphBatchSlots& S, cudaStream_t s)
{
    int nmax = 0;
    for (int i = 0; i < S.count; ++i) nmax = std::max(nmax, S.slot[i].n);
    if (S.count <= 0 || nmax <= 0) return cudaSuccess;
    k_merge_tails_group<<<dim3(2 * nmax, S.count), kMergeThreads, 0, s>>>(S);
    return cudaGetLastError();
}

cudaError_t launch_remove(sbc_graph* g, int u, int v, bool directed, int* d_res)
{
    k_remove<<<1, 32, 0, g->stream>>>(g->nv, g->d_row, g->d_deg, g->d_deg0, g->d_nsort, g->d_col, g->d_seq, u, v,
                                      directed ? 1 : 0, d_res);
    cudaError_t e = cudaGetLastError();
    if (e) return e;
    return launch_l2mask_remove(g, u, v, directed, d_res);
}

cudaError_t launch_mark_removed(sbc_graph* g, int n)
{
    if (n <= 0) return cudaSuccess;
    k_mark_removed<<<(int)(((int64_t)n * 32 + 127) / 128), 128, 0, g->stream>>>(g->d_row, g->d_deg, g->d_nsort, g->d_col, g->d_seq, n, g->d_ins,
                                           g->d_ins + g->ins_capacity, g->d_ins + 2 * g->ins_capacity);
    return cudaGetLastError();
}

cudaError_t launch_compact_removed(sbc_graph* g, int n)
{
    if (n <= 0) return cudaSuccess;
    k_compact_removed<<<2 * n, 256, 0, g->stream>>>(g->d_row, g->d_deg, g->d_deg0, g->d_nsort, g->d_col, g->d_seq, n,
                                                    g->d_ins, g->d_ins + g->ins_capacity,
                                                    g->d_ins + 2 * g->ins_capacity);
    cudaError_t e = cudaGetLastError();
    if (e) return e;
    if (n > 1) {
        k_reopen<<<(n + 255) / 256, 256, 0, g->stream>>>(g->d_deg, g->d_deg0, n, g->d_ins, g->d_ins + g->ins_capacity,
                                                         g->d_ins + 2 * g->ins_capacity);
        if ((e = cudaGetLastError())) return e;
    }
    return launch_l2mask_remove_batch(g, n);
}

cudaError_t launch_repack(sbc_graph* g, const int64_t* d_new_row, int32_t* d_new_col, int32_t* d_new_seq)
{
    int64_t blocks = (g->nv * 32 + 255) / 256;
    if (blocks > 152 * 64) blocks = 152 * 64;
    if (blocks < 1) blocks = 1;
    k_repack<<<(int)blocks, 256, 0, g->stream>>>(g->nv, g->d_row, g->d_deg, g->d_col, g->d_seq, d_new_row, d_new_col,
                                                 d_new_seq);
    return cudaGetLastError();
}

}  // namespace sbc
