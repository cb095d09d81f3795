// gtc_build.cuh -- kernels that orient the graph: degrees, the core's
// positions, the forward lists and the core's bit matrix.
#pragma once

#include <cooperative_groups.h>
#include <cooperative_groups/scan.h>

#include "gtc_internal.cuh"

namespace gtc {

namespace cg = cooperative_groups;

// What the kernels of one count read and write.
struct Data {
    const int *ind;                 // neighbour ids, graph-local in a batch
    long long n, nnz;
    const long long *vstart;        // batch: vertex starts, else null
    long long graphs;
    GraphRec *recs;
    unsigned int *hist;             // kBuckets per graph; counts, then cursors
    int *key;                       // degree, or kKeyTop - position for core vertices
    int *gid;                       // batch: graph of a vertex
    VInfo *vinfo;
    int *find;                      // forward lists; core members as -1 - position
    int *wide;                      // rows that blocks take
    int2 *litem;                    // placement items of long rows: {row, chunk}
    unsigned int *u;                // bit matrices
    long long ucap;                 // words of it
    unsigned long long *tacc;       // t(v) without the core's credits (null: global count only)
    unsigned long long *tcore;      // credits of core vertices: [first vertex + position]
    unsigned long long *gsum;       // batch: sum of t per graph
    Counters *ctr;
    unsigned int *status;
    int word;                       // sizeof(unsigned int)
};
template <typename OffT>
struct View : Data {
    const OffT *off;
};

template <typename OffT>
__device__ __forceinline__ int row_degree(const View<OffT> &w, long long v)
{
    return (int)((long long)w.off[v + 1] - (long long)w.off[v]);
}

// Graph holding vertex v: the largest g < G with vstart[g] <= v.
__device__ __forceinline__ int graph_of(const long long *__restrict__ vstart, long long G,
                                        long long v)
{
    long long lo = 0, hi = G;
    while (hi - lo > 1) {
        const long long mid = (lo + hi) >> 1;
        if (vstart[mid] <= v) lo = mid; else hi = mid;
    }
    return (int)lo;
}

// A graph's limits: the lowest degree that may be core, the longest row that
// is not posted as a long row, the most core vertices.  The core is worth its
// bit matrix where degrees are skewed: a vertex of at least kCoreDegreeRatio
// times the mean degree (uniform graphs have none, so they pay nothing but
// the empty launches).  A small graph so dense that its whole bit matrix is
// no larger than its adjacency lists (mean degree >= n / 32) is all core.
__host__ __device__ __forceinline__ void core_limits(long long n, long long nnz, long long room,
                                                     int &dmin, int &long_min, int &kcap)
{
    const bool all = n <= room && n <= kCoreMax && n * n <= 32 * nnz;
    const long long least = div_up<long long>(kCoreDegreeRatio * nnz, n > 0 ? n : 1);
    dmin = all ? 1 : (int)(least > kCoreMinDegree ? least : kCoreMinDegree);
    long_min = all ? 0 : kShortRow;
    const long long most = all ? n : n / 4;
    kcap = (int)(most < room ? most : room);
}

// Core rows that a batch graph of n vertices has room for: its bit matrix
// takes at most 64 bytes per vertex.
__device__ __forceinline__ long long batch_room(long long n)
{
    if (n <= 768) return n;
    const long long k = (long long)(30.0f * sqrtf((float)n));
    return k < kCoreMax ? k : kCoreMax;
}

// Batch, one thread per graph: the limits and the vertex range.
template <typename OffT>
__device__ __forceinline__ GraphRec batch_limits(const View<OffT> &w, long long g)
{
    GraphRec r;
    r.v0 = w.vstart[g];
    r.nv = (int)(w.vstart[g + 1] - r.v0);
    const long long nnz = (long long)w.off[r.v0 + r.nv] - (long long)w.off[r.v0];
    core_limits(r.nv, nnz, batch_room(r.nv), r.dmin, r.long_min, r.kcap);
    return r;
}

template <typename OffT>
__global__ void graph_limits_kernel(const View<OffT> w)
{
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g < w.graphs) w.recs[g] = batch_limits(w, g);
}

// gid[v] of a batch; a block finds its first vertex's graph, threads walk on.
template <typename OffT>
__device__ __forceinline__ int walk_graph(const View<OffT> &w, long long v, int g)
{
    while (g + 1 < w.graphs && w.vstart[g + 1] <= v) ++g;
    return g;
}

template <typename OffT>
__global__ void graph_ids_kernel(const View<OffT> w)
{
    __shared__ int s_g;
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (threadIdx.x == 0) s_g = graph_of(w.vstart, w.graphs, v);
    __syncthreads();
    if (v < w.n) w.gid[v] = walk_graph(w, v, s_g);
}

// Choose a graph's core from its degree histogram (one block of kThreads): the
// most top buckets that fit kcap.  hist becomes the buckets' first positions.
__device__ __forceinline__ void choose_core(unsigned int *hist, int dmin, int kcap,
                                            int &min_bucket, int &core)
{
    constexpr int kPer = kBuckets / kThreads;
    __shared__ unsigned int s_sum[kThreads / 32];
    __shared__ int s_min, s_core;
    // thread t holds the buckets top - t * kPer - j, j < kPer: a prefix in
    // descending degree
    const int top = kBuckets - 1 - (int)threadIdx.x * kPer;
    unsigned int h[kPer], mine = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        h[j] = __ldcg(&hist[top - j]);
        mine += h[j];
    }
    if (threadIdx.x == 0) { s_min = kBuckets; s_core = 0; }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
    }
    if (lane == 31) s_sum[warp] = incl;
    __syncthreads();
    unsigned int run = incl - mine;
    for (int i = 0; i < warp; ++i) run += s_sum[i];
    const int bmin = degree_bucket(dmin);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        hist[top - j] = run;
        run += h[j];
        if (top - j >= bmin && run <= (unsigned int)kcap) {
            atomicMin(&s_min, top - j);
            atomicMax(&s_core, (int)run);
        }
    }
    __syncthreads();
    core = s_core;
    min_bucket = core > 0 ? s_min : kBuckets;
}

// Long row i of the wide list: its record, its placement items and, for a
// core vertex, its key.
template <typename OffT>
__device__ __forceinline__ void key_row(const View<OffT> &w, long long i)
{
    const int v = __ldcg(&w.wide[i]);
    const long long b = (long long)w.off[v];
    const int d = (int)((long long)w.off[v + 1] - b);
    const int g = w.vstart ? w.gid[v] : 0;
    w.vinfo[v] = VInfo{b, 0, kWideRow};
    const int bk = degree_bucket(d);
    if (bk >= w.recs[g].min_bucket)
        w.key[v] = kKeyTop - (int)atomicAdd(&w.hist[(long long)g * kBuckets + bk], 1u);
    // one reservation per group of converged lanes
    const int k = div_up(d, kRowChunk);
    auto grp = cg::coalesced_threads();
    const int incl = cg::inclusive_scan(grp, k);
    const int last = (int)grp.size() - 1;
    unsigned long long at = 0;
    if ((int)grp.thread_rank() == last)
        at = atomicAdd(&w.ctr->place_items, (unsigned long long)incl);
    at = grp.shfl(at, last) + (unsigned long long)(incl - k);
    for (int c = 0; c < k; ++c) w.litem[at + c] = make_int2(v, c);
}

// Degrees: key[v] = d(v), the histogram of the degrees that may be core, and
// the list of long rows.  With `choose` (single graph) the last block to
// finish chooses the core, which saves a launch; with `ids` (batch) the graph
// ids and limits are found here too.
template <typename OffT, bool BATCH>
__global__ void __launch_bounds__(kThreads)
degree_kernel(const View<OffT> w, GraphRec lim, bool ids, bool choose)
{
    __shared__ int s_g;
    __shared__ bool s_last;
    const long long v = (long long)blockIdx.x * kThreads + threadIdx.x;
    if (BATCH && ids) {
        if (threadIdx.x == 0) s_g = graph_of(w.vstart, w.graphs, v < w.n ? v : w.n - 1);
        __syncthreads();
    }
    bool lng = false;
    if (v < w.n) {
        const int d = row_degree(w, v);
        w.key[v] = d;
        int g = 0;
        if (BATCH) {
            if (ids) {
                g = walk_graph(w, v, s_g);
                w.gid[v] = g;
                lim = batch_limits(w, g);
            } else {
                g = w.gid[v];
                lim = w.recs[g];
            }
        }
        lng = d > lim.long_min;
        const int bk = degree_bucket(d);
        if (lng && bk >= degree_bucket(lim.dmin))
            atomicAdd(&w.hist[(long long)g * kBuckets + bk], 1u);
    }
    const unsigned int m = __ballot_sync(0xffffffffu, lng);
    const int lane = threadIdx.x & 31;
    if (m) {
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(&w.ctr->wide_rows, (unsigned long long)__popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (lng) w.wide[at + __popc(m & ((1u << lane) - 1u))] = (int)v;
    }
    if (!choose) return;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&w.ctr->blocks_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    choose_core(w.hist, lim.dmin, lim.kcap, lim.min_bucket, lim.core);
    if (threadIdx.x == 0) w.recs[0] = lim;
}

// One block per graph: its core, and its share of the bit-matrix words.
template <typename OffT, bool BATCH>
__global__ void __launch_bounds__(kThreads)
choose_core_kernel(const View<OffT> w, GraphRec lim, bool limits)
{
    const long long g = blockIdx.x;
    if (BATCH) lim = limits ? batch_limits(w, g) : w.recs[g];
    int min_bucket = 0, core = 0;
    choose_core(w.hist + g * kBuckets, lim.dmin, lim.kcap, min_bucket, core);
    if (threadIdx.x == 0) {
        lim.min_bucket = min_bucket;
        lim.core = core;
        if (BATCH && core > 0) {
            const unsigned long long words = (unsigned long long)u_row(core);
            lim.ubase = (long long)atomicAdd(&w.ctr->u_words, words);
            if (lim.ubase + (long long)words > w.ucap) {     // no room: no core
                lim.core = 0;
                lim.min_bucket = kBuckets;
                lim.ubase = 0;
            }
        }
        w.recs[g] = lim;
    }
}

// Bit-matrix words in use, all graphs.
__device__ __forceinline__ long long u_words(const Data &w)
{
    const long long k = w.vstart ? (long long)w.ctr->u_words : (long long)u_row(w.recs[0].core);
    return k < w.ucap ? k : w.ucap;
}

__device__ __forceinline__ void zero_bits(const Data &w)
{
    const long long quads = u_words(w) / 4;          // u_row is a multiple of 8
    uint4 *q = reinterpret_cast<uint4 *>(w.u);
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < quads; i += stride)
        q[i] = make_uint4(0u, 0u, 0u, 0u);
}

__global__ void zero_bits_kernel(const Data w)
{
    zero_bits(w);
}

template <typename OffT>
__global__ void key_rows_kernel(const View<OffT> w, bool zero)
{
    if (zero) zero_bits(w);
    const long long rows = (long long)w.ctr->wide_rows;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += stride)
        key_row(w, i);
}

// Forward lists, and the core's bit-matrix rows, in one pass over the
// adjacency.  x is above v when its key is (ties: the larger id).
//   * long rows, a block per kRowChunk entries, eight per thread with all
//     gathers of keys in flight; members are appended a warp's at a time, at
//     positions reserved by one 64-bit add on {fdeg, dk}, and a core row sets
//     its bits;
//   * the other rows, a thread each, four entries at a time.  Their lists
//     start at a multiple of four entries where the row leaves room, for
//     16-byte loads.
// The order within a list is arbitrary.
template <typename OffT, bool BATCH>
__device__ __forceinline__ void place_chunk(const View<OffT> &w, int2 it)
{
    constexpr int kPer = kRowChunk / kThreads;
    const int v = it.x;
    const long long b = (long long)w.off[v], e = (long long)w.off[v + 1];
    const long long s = b + (long long)it.y * kRowChunk;
    const int kv = w.key[v];
    long long v0 = 0, nv = w.n, ubase = 0;
    int g = 0;
    if (BATCH) g = w.gid[v];
    const GraphRec *rec = &w.recs[g];
    if (BATCH) { v0 = rec->v0; nv = rec->nv; ubase = rec->ubase; }
    const int kmin = kKeyTop - rec->core;            // keys above it are core
    int x[kPer], kx[kPer];
    bool bad = false;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const long long i = s + j * kThreads + threadIdx.x;
        x[j] = i < e ? w.ind[i] : -1;
        const bool ok = (unsigned long long)(long long)x[j] < (unsigned long long)nv;
        bad |= i < e && !ok;
        x[j] = ok ? (int)(x[j] + v0) : -1;
    }
#pragma unroll
    for (int j = 0; j < kPer; ++j) kx[j] = x[j] >= 0 ? w.key[x[j]] : -1;
    if (bad) atomicOr(w.status, kErrIndexRange);
    if (kv > kmin) {
        unsigned int *row = w.u + ubase + u_row(kKeyTop - kv);
#pragma unroll
        for (int j = 0; j < kPer; ++j)
            if (kx[j] > kv) {
                const int pos = kKeyTop - kx[j];
                atomicOr(&row[pos >> 5], 1u << (pos & 31));
            }
    }
    const int lane = threadIdx.x & 31;
    unsigned int fwd[kPer];
    int total = 0, dk = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const bool f = kx[j] > kv || (kx[j] == kv && x[j] > v);
        fwd[j] = __ballot_sync(0xffffffffu, f);
        total += __popc(fwd[j]);
        dk += __popc(__ballot_sync(0xffffffffu, f && kx[j] > kmin));
    }
    if (total == 0) return;
    unsigned long long at = 0;
    if (lane == 0)
        at = atomicAdd(reinterpret_cast<unsigned long long *>(&w.vinfo[v].fdeg),
                       (unsigned long long)total | ((unsigned long long)dk << 32));
    int p = (int)(unsigned int)__shfl_sync(0xffffffffu, at, 0);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        if ((fwd[j] >> lane) & 1u)
            w.find[b + p + __popc(fwd[j] & ((1u << lane) - 1u))] =
                kx[j] > kmin ? (int)((unsigned int)kx[j] ^ 0x80000000u) : x[j];
        p += __popc(fwd[j]);
    }
}

template <typename OffT, bool BATCH>
__device__ __forceinline__ void place_short(const View<OffT> &w, long long v)
{
    if (v >= w.n) return;
    const long long b = (long long)w.off[v];
    const int d = (int)((long long)w.off[v + 1] - b);
    const GraphRec *rec = &w.recs[BATCH ? w.gid[v] : 0];
    if (d > rec->long_min) return;
    const int v0 = BATCH ? (int)rec->v0 : 0;
    const unsigned int nv = BATCH ? (unsigned int)rec->nv : (unsigned int)w.n;
    const int kmin = kKeyTop - rec->core;
    int *list = w.find + b;
    int start = (int)(-b & 3), wrote = 0, dk = 0;
    if (start >= d) start = 0;
    bool bad = false;
    for (int k = 0; k < d; k += 4) {
        int x[4], kx[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = k + j < d ? w.ind[b + k + j] : -1;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const bool ok = (unsigned int)x[j] < nv;
            bad |= !ok && k + j < d;
            x[j] += v0;
            kx[j] = ok ? w.key[x[j]] : -1;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (kx[j] > d || (kx[j] == d && x[j] > v)) {
                const bool core = kx[j] > kmin;
                if (start > 0 && start + wrote == d) {      // no room: to the row's begin
                    for (int i = 0; i < wrote; ++i) list[i] = list[start + i];
                    start = 0;
                }
                list[start + wrote++] = core ? (int)((unsigned int)kx[j] ^ 0x80000000u) : x[j];
                dk += core;
            }
    }
    if (bad) atomicOr(w.status, kErrIndexRange);
    if (wrote > kShortList) {
        dk |= kWideRow;
        w.wide[atomicAdd(&w.ctr->wide_rows, 1ull)] = (int)v;
    }
    w.vinfo[v] = VInfo{b + start, wrote, dk};
}

template <typename OffT, bool BATCH>
__global__ void __launch_bounds__(kThreads)
place_kernel(const View<OffT> w, bool do_wide, bool do_short)
{
    __shared__ long long s_item;
    // a block's first item is its own index, the next ones come from a queue
    auto items = [&](unsigned long long *queue, long long n, const auto &item) {
        long long i = blockIdx.x;
        while (i < n) {
            item(i);
            if (gridDim.x >= n) break;
            __syncthreads();
            if (threadIdx.x == 0) s_item = (long long)atomicAdd(queue, 1ull) + gridDim.x;
            __syncthreads();
            i = s_item;
        }
    };
    if (do_wide)
        items(&w.ctr->place_next, (long long)w.ctr->place_items,
              [&](long long i) { place_chunk<OffT, BATCH>(w, w.litem[i]); });
    if (do_short)
        items(&w.ctr->tile_next, div_up<long long>(w.n, kThreads),
              [&](long long i) { place_short<OffT, BATCH>(w, i * kThreads + threadIdx.x); });
}

}  // namespace gtc
