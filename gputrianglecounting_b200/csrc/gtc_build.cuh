// gtc_build.cuh -- kernels that orient the graph: degrees, the core's
// positions, the forward lists and the core's bit matrix.
#pragma once

#include <cooperative_groups.h>
#include <cooperative_groups/scan.h>

#include "gtc_data.cuh"

namespace gtc {

namespace cg = cooperative_groups;

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
// bit matrix where degrees are skewed: a vertex of at least twice the mean
// degree and 16 more, which random graphs of equal expected degrees do not have
// (eight standard deviations at mean 32), so those stay uniform and pay nothing
// but the empty launches.  At 4 and 8 times the mean the 512-graph batch took
// 10.64 and 12.31 ms instead of 10.37, R-MAT 17 181 and 200 us instead of 170.
// A small graph of mean degree 64 or more, so dense that its whole bit matrix is
// no larger than its adjacency lists (mean degree >= n / 32), is all core.
__host__ __device__ __forceinline__ void core_limits(long long n, long long nnz, long long room,
                                                     int &dmin, int &long_min, int &kcap)
{
    const bool all = n <= room && n <= kCoreMax && n * n <= 32 * nnz && nnz >= 64 * n;
    const long long least =
        kCoreDegreeOver + div_up<long long>(kCoreDegreeRatio * nnz, n > 0 ? n : 1);
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
                                            int &min_bucket, int &core, int &uniform)
{
    constexpr int kPer = kBuckets / kThreads;
    __shared__ unsigned int s_sum[kThreads / 32];
    __shared__ int s_min, s_core, s_any;
    // thread t holds the buckets top - t * kPer - j, j < kPer: a prefix in
    // descending degree
    const int top = kBuckets - 1 - (int)threadIdx.x * kPer;
    unsigned int h[kPer], mine = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        h[j] = __ldcg(&hist[top - j]);
        mine += h[j];
    }
    if (threadIdx.x == 0) { s_min = kBuckets; s_core = 0; s_any = 0; }
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
        if (h[j]) s_any = 1;
        if (top - j >= bmin && run <= (unsigned int)kcap) {
            atomicMin(&s_min, top - j);
            atomicMax(&s_core, (int)run);
        }
    }
    __syncthreads();
    core = s_core;
    min_bucket = core > 0 ? s_min : kBuckets;
    uniform = !s_any;
}

// Whether a uniform graph's rows get signatures (one block): where they fit in
// the graph's part of find, which such a graph leaves unused, and less than a
// twelfth of sampled pairs of neighbours are neighbours themselves.  A pair
// that the signature lets pass is searched for, so signatures pay where most
// pairs are none; where many are edges, tiles of rows share members and do
// better.  Place and list kernels, signatures and tiles: 524K vertices of mean
// degree 30, no closed pairs 180 and 324 us, 4% 232 and 325, 15% 398 and 295,
// 58% 1124 and 201; of mean degree 16, 4% 112 and 151, 15% 151 and 138.  The
// sample costs 5 us, which calls of few vertices do not earn back (ER 16K: list
// kernel 14.7 -> 11.8 us, degree kernel 4.4 -> 8.6).
template <typename OffT>
__device__ __forceinline__ bool use_signatures(const View<OffT> &w, GraphRec &rec)
{
    constexpr int kPer = 4;                          // samples per warp, in flight together
    __shared__ int s_seen, s_closed;
    const long long first = (long long)w.off[rec.v0], last = (long long)w.off[rec.v0 + rec.nv];
    const long long base = div_up<long long>(first, kSigWords) * kSigWords;
    if (w.n < kSignedCall || rec.nv < kSignedGraph ||
        base + (long long)kSigWords * rec.nv > last)
        return false;
    if (threadIdx.x == 0) s_seen = s_closed = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    long long b[kPer], d[kPer];
    int y[kPer];
    unsigned int h[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        h[j] = (unsigned int)((threadIdx.x >> 5) * kPer + j + 1) * 0x9E3779B1u;
        const long long v = rec.v0 + (((unsigned long long)h[j] * (unsigned int)rec.nv) >> 32);
        b[j] = (long long)w.off[v];
        d[j] = (long long)w.off[v + 1] - b[j];
    }
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const bool pair = d[j] >= 2;
        const unsigned int i = pair ? h[j] % (unsigned int)(d[j] - 1) : 0u;
        const unsigned int k = pair ? i + 1 + (h[j] >> 7) % (unsigned int)(d[j] - 1 - i) : 0u;
        const int x = pair ? w.ind[b[j] + i] : -1;
        y[j] = pair ? w.ind[b[j] + k] : -1;
        const bool in = (unsigned int)x < (unsigned int)rec.nv;
        b[j] = in ? (long long)w.off[rec.v0 + x] : 0;
        d[j] = in ? (long long)w.off[rec.v0 + x + 1] - b[j] : -1;
    }
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        bool hit = false;
        for (long long i = lane; i < d[j]; i += 32) hit |= w.ind[b[j] + i] == y[j];
        hit = __any_sync(0xffffffffu, hit);
        if (lane == 0 && d[j] >= 0) {
            atomicAdd(&s_seen, 1);
            if (hit) atomicAdd(&s_closed, 1);
        }
    }
    __syncthreads();
    const bool yes = 12 * s_closed < s_seen;
    if (yes) rec.ubase = base;
    return yes;
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
    if (w.recs[g].uniform) return;
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
__global__ void __launch_bounds__(kThreads, 8)
degree_kernel(const View<OffT> w, GraphRec lim, bool ids, bool choose)
{
    if (gated(w)) return;
    __shared__ int s_g;
    __shared__ bool s_last;
    __shared__ unsigned int s_hist[BATCH ? 1 : kBuckets];
    const int lane = threadIdx.x & 31;
    const long long stride = (long long)gridDim.x * kThreads;
    // a large graph's blocks count for themselves first: the buckets of the
    // lowest core degrees are many vertices' (R-MAT 22: 105 us, 42 so)
    const bool own = !BATCH && w.n > stride;
    if (own) {
        for (int k = threadIdx.x; k < kBuckets; k += kThreads) s_hist[k] = 0;
        __syncthreads();
    }
    for (long long v0 = (long long)blockIdx.x * kThreads; v0 < w.n; v0 += stride) {
        const long long v = v0 + threadIdx.x;
        if (BATCH && ids) {
            __syncthreads();
            if (threadIdx.x == 0) s_g = graph_of(w.vstart, w.graphs, v0);
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
                atomicAdd(own ? &s_hist[BATCH ? 0 : bk] : &w.hist[(long long)g * kBuckets + bk], 1u);
        }
        const unsigned int m = __ballot_sync(0xffffffffu, lng);
        if (m) {
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(&w.ctr->wide_rows, (unsigned long long)__popc(m));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (lng) w.wide[at + __popc(m & ((1u << lane) - 1u))] = (int)v;
        }
    }
    if (own) {
        __syncthreads();
        for (int k = threadIdx.x; k < kBuckets; k += kThreads)
            if (s_hist[k]) atomicAdd(&w.hist[k], s_hist[k]);
    }
    if (BATCH || !choose) return;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&w.ctr->blocks_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    choose_core(w.hist, lim.dmin, lim.kcap, lim.min_bucket, lim.core, lim.uniform);
    if (lim.uniform && use_signatures(w, lim)) lim.uniform = kSigned;
    if (threadIdx.x == 0) w.recs[0] = lim;
}

// A graph's core, by the block, and its share of the bit-matrix words.
template <typename OffT, bool BATCH>
__device__ __forceinline__ void choose_graph_core(const View<OffT> &w, long long g, GraphRec lim)
{
    int min_bucket = 0, core = 0, uniform = 0;
    choose_core(w.hist + g * kBuckets, lim.dmin, lim.kcap, min_bucket, core, uniform);
    if (uniform && use_signatures(w, lim)) uniform = kSigned;
    if (threadIdx.x == 0) {
        lim.uniform = uniform;
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

// The cores of `per` graphs per block.  A thread settles a graph of no more
// vertices than a short row has entries, which has no core and no signatures,
// so that a batch of many tiny graphs does not pay a block and a look at an
// empty histogram for each (100,000 graphs of 16 vertices: the count takes 314
// us, with a block for each 729).
template <typename OffT, bool BATCH>
__global__ void __launch_bounds__(kThreads)
choose_core_kernel(const View<OffT> w, GraphRec lim, bool limits, int per)
{
    auto limits_of = [&](long long g) { return limits ? batch_limits(w, g) : w.recs[g]; };
    if (!BATCH || per == 1) {
        choose_graph_core<OffT, BATCH>(w, blockIdx.x, BATCH ? limits_of(blockIdx.x) : lim);
        return;
    }
    __shared__ int s_todo[kThreads], s_n;
    const long long g0 = (long long)blockIdx.x * per;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    if (threadIdx.x < per && g0 + threadIdx.x < w.graphs) {
        lim = limits_of(g0 + threadIdx.x);
        if (lim.nv <= lim.long_min) {
            lim.uniform = 1;
            w.recs[g0 + threadIdx.x] = lim;
        } else {
            s_todo[atomicAdd(&s_n, 1)] = (int)threadIdx.x;
        }
    }
    __syncthreads();
    for (int k = 0; k < s_n; ++k) {
        const long long g = g0 + s_todo[k];
        choose_graph_core<OffT, BATCH>(w, g, limits_of(g));
        __syncthreads();                          // its shared words are used again
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
    if (gated(w)) return;
    if (zero) zero_bits(w);
    const long long rows = (long long)w.ctr->wide_rows;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += stride)
        key_row(w, i);
}

// Where the rows of a graph keep their forward lists, and what turns a list's
// ids into vertices: a uniform graph's rows are ordered by id, so a forward
// list is the end of the row itself.
struct Lists {
    const int *base;
    int shift;
};

template <bool BATCH>
__device__ __forceinline__ Lists lists_of(const Data &w, const GraphRec *rec)
{
    return rec->uniform ? Lists{w.ind, BATCH ? (int)rec->v0 : 0} : Lists{w.find, 0};
}

// Forward lists, and the core's bit-matrix rows, in one pass over the
// adjacency.  x is above v when its key is (ties: the larger id).
//   * long rows, kRowChunk entries per warp, eight per lane with all gathers of
//     keys in flight; members are appended at positions reserved by one 64-bit
//     add on {fdeg, dk}, and a core row sets its bits;
//   * the other rows, 32 consecutive ones per warp, their entries as one
//     stream, 128 at a time;
//   * rows of a uniform graph (no degree above a few times the mean) are
//     ordered by id: no keys are gathered and no list is written, only where
//     the ids above the row's begin.
// The order within a list is arbitrary.  The gathers of keys, from L2, bound it,
// four to eight in flight per lane: R-MAT 20 166 us (merge-path tiles with a sort
// of the lists 480), RGG 4M 93 (185), the 512-graph batch 1675 (3308).
template <typename OffT, bool BATCH>
__device__ __forceinline__ void place_chunk(const View<OffT> &w, int2 it)
{
    constexpr int kPer = kRowChunk / 32;
    const int lane = threadIdx.x & 31;
    const int v = it.x;
    const long long b = (long long)w.off[v], e = (long long)w.off[v + 1];
    const long long s = b + (long long)it.y * kRowChunk;
    const int kv = w.key[v];
    const GraphRec *rec = &w.recs[BATCH ? w.gid[v] : 0];
    const int v0 = BATCH ? (int)rec->v0 : 0;
    const unsigned int nv = BATCH ? (unsigned int)rec->nv : (unsigned int)w.n;
    const int kmin = kKeyTop - rec->core;            // keys above it are core
    int x[kPer], kx[kPer];
    bool bad = false;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const long long i = s + j * 32 + lane;
        x[j] = i < e ? w.ind[i] : 0;
        const bool ok = (unsigned int)x[j] < nv;
        bad |= !ok;
        x[j] = i < e && ok ? x[j] + v0 : -1;
    }
#pragma unroll
    for (int j = 0; j < kPer; ++j) kx[j] = x[j] >= 0 ? w.key[x[j]] : -1;
    if (bad) atomicOr(w.status, kErrIndexRange);
    if (kv > kmin) {
        unsigned int *row = w.u + (BATCH ? rec->ubase : 0) + u_row(kKeyTop - kv);
#pragma unroll
        for (int j = 0; j < kPer; ++j)
            if (kx[j] > kv) {
                const int pos = kKeyTop - kx[j];
                atomicOr(&row[pos >> 5], 1u << (pos & 31));
            }
    }
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

// Lanes [lo, hi) as a mask; empty for hi <= lo.
__device__ __forceinline__ unsigned int lane_range(int lo, int hi)
{
    lo = max(lo, 0);
    hi = min(hi, 32);
    return hi > lo ? (0xffffffffu >> (32 - hi)) & (0xffffffffu << lo) : 0u;
}

// A placed row's record; a list longer than `most` makes it a wide row.
__device__ __forceinline__ void row_record(const Data &w, long long v, long long fbeg, int fdeg,
                                           int dk, int most, bool listed)
{
    if (!listed && fdeg > most) w.wide[atomicAdd(&w.ctr->wide_rows, 1ull)] = (int)v;
    if (listed || fdeg > most) dk |= kWideRow;
    w.vinfo[v] = VInfo{fbeg, fdeg, dk};
}

// The signatures of 32 rows, a lane each: bits[word][lane].
typedef unsigned int SignSmem[kSigWords][32];

// Of the first `rows` rows from u0 on, those of uniform graphs (mine): where the ids
// above the row's own begin (b, e: the lane's row), and the signature of those ids.
template <typename OffT, bool BATCH, bool SIGN>
__device__ __forceinline__ void split_rows(const View<OffT> &w, long long u0, int rows, int g, bool mine,
                                           long long b, long long e, SignSmem &bits)
{
    const int lane = threadIdx.x & 31;
    const long long v = u0 + lane;
    int vl = 0, long_min = 0;
    unsigned int nv = 0;
    unsigned int *sign = nullptr;
    if (mine) {
        const GraphRec *rec = &w.recs[g];
        if (SIGN && rec->uniform == kSigned)
            sign = reinterpret_cast<unsigned int *>(w.find) + rec->ubase +
                   kSigWords * (v - (BATCH ? rec->v0 : 0));
        nv = BATCH ? (unsigned int)rec->nv : (unsigned int)w.n;
        vl = (int)(v - (BATCH ? rec->v0 : 0));
        long_min = rec->long_min;
    }
    // ids out of range, looked for in the rows' entries as one stream
    bool bad = false;
    const int g0 = __shfl_sync(0xffffffffu, g, 0);
    if (__all_sync(0xffffffffu, lane >= rows || (mine && g == g0))) {
        const unsigned int n0 = __shfl_sync(0xffffffffu, nv, 0);
        const long long b0 = __shfl_sync(0xffffffffu, b, 0);
        const long long e1 = __shfl_sync(0xffffffffu, e, rows - 1);
        for (long long i = b0 + lane; i < e1; i += 128) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (i + 32 * j < e1) bad |= (unsigned int)w.ind[i + 32 * j] >= n0;
        }
    } else {
        bad = true;                               // each lane looks at its own row
    }
    if (__any_sync(0xffffffffu, bad)) {
        bad = false;
        for (long long i = b; i < e; ++i) bad |= (unsigned int)w.ind[i] >= nv;
        if (bad) atomicOr(w.status, kErrIndexRange);
    }
    if (!mine) return;
    const bool listed = (int)(e - b) > long_min;
    long long lo = b;
    if (bad) {
        // ids out of range are first or last in the row
        while (lo < e && !((unsigned int)w.ind[lo] < nv && w.ind[lo] > vl)) ++lo;
        for (long long i = lo; i < e; ++i)
            if ((unsigned int)w.ind[i] >= nv) e = i;
    }
    int len = bad ? 0 : (int)(e - b);
    while (len > 0) {
        const int half = len >> 1;
        if (w.ind[lo + half] <= vl) {
            lo += half + 1;
            len -= half + 1;
        } else {
            len = half;
        }
    }
    row_record(w, v, lo, e > lo ? (int)(e - lo) : 0, 0, kShortListIds, listed);
    if constexpr (SIGN) {
        if (!sign) return;
#pragma unroll
        for (int k = 0; k < kSigWords; ++k) bits[k][lane] = 0;
        const int *list = w.ind + lo;
        const int n = (int)(e - lo);
        for (int i = 0; i < n; i += 4) {
            int y[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] = list[min(i + j, n - 1)];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const Sign x = sign_of(y[j]);
                bits[x.word][lane] |= x.bits;
            }
        }
        uint4 *to = reinterpret_cast<uint4 *>(sign);
        to[0] = make_uint4(bits[0][lane], bits[1][lane], bits[2][lane], bits[3][lane]);
        to[1] = make_uint4(bits[4][lane], bits[5][lane], bits[6][lane], bits[7][lane]);
    }
}

// Of the first `rows` rows from u0 on, those of other graphs that are not long rows.
template <typename OffT, bool BATCH>
__device__ __forceinline__ void stream_rows(const View<OffT> &w, long long u0, int rows, int g)
{
    constexpr int kPer = 4;
    const int lane = threadIdx.x & 31;
    const long long v = u0 + lane;
    long long b = 0;
    int d = 0, kmin = kKeyTop, v0 = 0, nv = (int)w.n;
    bool mine = false;
    if (lane < rows) {
        const GraphRec *rec = &w.recs[g];
        b = (long long)w.off[v];
        d = (int)((long long)w.off[v + 1] - b);
        mine = !rec->uniform && d <= rec->long_min;
        kmin = kKeyTop - rec->core;
        if (BATCH) {
            v0 = (int)rec->v0;
            nv = rec->nv;
        }
    }
    const int n = mine && d > 0 ? d : 0;
    const int incl = warp_incl_scan(n), excl = incl - n;
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    const long long start = b - excl;
    int wrote = 0, dk = 0;
    bool bad = false;
    for (int f0 = 0; f0 < total; f0 += 32 * kPer) {
        int i[kPer], x[kPer], kx[kPer];
        long long at[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int f = f0 + 32 * j + lane;
            i[j] = warp_corank(incl, f);
            at[j] = __shfl_sync(0xffffffffu, start, i[j]);
            x[j] = f < total ? w.ind[at[j] + f] : 0;
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int f = f0 + 32 * j + lane;
            const int nj = BATCH ? __shfl_sync(0xffffffffu, nv, i[j]) : nv;
            const int vj = BATCH ? __shfl_sync(0xffffffffu, v0, i[j]) : 0;
            const bool ok = (unsigned int)x[j] < (unsigned int)nj;
            bad |= !ok;
            x[j] = f < total && ok ? x[j] + vj : -1;
            kx[j] = x[j] >= 0 ? w.key[x[j]] : -1;
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int g0 = f0 + 32 * j;
            if (g0 >= total) break;
            const int di = __shfl_sync(0xffffffffu, d, i[j]);
            const int ki = __shfl_sync(0xffffffffu, kmin, BATCH ? i[j] : 0);
            const int ei = __shfl_sync(0xffffffffu, excl, i[j]);
            const int wi = __shfl_sync(0xffffffffu, wrote, i[j]);
            const bool f = kx[j] > di || (kx[j] == di && x[j] > (int)(u0 + i[j]));
            const bool core = kx[j] > ki;
            const unsigned int mf = __ballot_sync(0xffffffffu, f);
            const unsigned int mk = __ballot_sync(0xffffffffu, f && core);
            if (f) {
                // members of this row before this one: earlier steps', and
                // this step's from the row's first lane on
                const int p = wi + __popc(mf & lane_range(ei - g0, lane));
                w.find[at[j] + ei + p] = core ? (int)((unsigned int)kx[j] ^ 0x80000000u) : x[j];
            }
            const unsigned int own = lane_range(excl - g0, incl - g0);
            wrote += __popc(mf & own);
            dk += __popc(mk & own);
        }
    }
    if (bad) atomicOr(w.status, kErrIndexRange);
    if (mine) row_record(w, v, b, wrote, dk, kShortList, false);
}

template <typename OffT, bool BATCH>
__global__ void __launch_bounds__(kThreads, 5)
place_kernel(const View<OffT> w, bool do_wide, bool do_short, int batch)
{
    __shared__ SignSmem s_sign[kThreads / 32];
    if (gated(w)) return;
    const int lane = threadIdx.x & 31;
    const long long warps = (long long)gridDim.x * (kThreads / 32);
    const long long warp = (long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    if (do_wide) {
        // chunks are alike, so a fixed share of them is an even one
        const long long items = (long long)w.ctr->place_items;
        for (long long i = warp; i < items; i += warps) place_chunk<OffT, BATCH>(w, w.litem[i]);
    }
    if (!do_short) return;
    long long u0 = warp * batch;
    // the lane's row's entries, if it is `mine`; else none
    auto ends = [&](long long u, bool mine, long long &b, long long &e) {
        b = e = 0;
        if (mine && u + lane < w.n) {
            b = (long long)w.off[u + lane];
            e = (long long)w.off[u + lane + 1];
        }
    };
    if (!BATCH && w.recs[0].uniform && w.recs[0].uniform != kSigned) {
        // rows alike, so fixed shares are even ones, and the next share's
        // offsets can be on their way (RGG 4M 117 -> 95 us, of mean degree 4
        // 97 -> 56).  With signatures to build they are not: the lowest ids
        // have the longest lists (ER 900K 62 us from the queue, 79 so).
        long long b, e;
        ends(u0, lane < batch, b, e);
        while (u0 < w.n) {
            const long long u1 = u0 + warps * batch;
            const int rows = (int)min((long long)batch, w.n - u0);
            long long b1, e1;
            ends(u1, lane < batch, b1, e1);
            split_rows<OffT, BATCH, false>(w, u0, rows, 0, lane < rows, b, e,
                                    s_sign[threadIdx.x >> 5]);
            u0 = u1;
            b = b1;
            e = e1;
        }
        return;
    }
    while (u0 < w.n) {
        const int rows = (int)min((long long)batch, w.n - u0);
        const bool in = lane < rows;
        const int g = BATCH && in ? w.gid[u0 + lane] : 0;
        const bool uniform = in && w.recs[g].uniform;
        if (__any_sync(0xffffffffu, uniform)) {
            long long b, e;
            ends(u0, uniform, b, e);
            split_rows<OffT, BATCH, true>(w, u0, rows, g, uniform, b, e, s_sign[threadIdx.x >> 5]);
        }
        if (__any_sync(0xffffffffu, in && !uniform)) stream_rows<OffT, BATCH>(w, u0, rows, g);
        if (warps * batch >= w.n) break;
        if (lane == 0) u0 = batch * (warps + (long long)atomicAdd(&w.ctr->place_next, 1ull));
        u0 = __shfl_sync(0xffffffffu, u0, 0);
    }
}

}  // namespace gtc
