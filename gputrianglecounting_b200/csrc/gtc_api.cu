// gtc_api.cu -- the C ABI (include/gtc_b200.h): status strings, workspace
// sizing, the counting entry points, the CSR validator, the vertex-subset
// kernel and the reference-compatible kernelCall shims.
#include <cooperative_groups.h>
#include <cooperative_groups/reduce.h>

#include <climits>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "gtc_core.cuh"
#include "gtc_data.cuh"

namespace cg = cooperative_groups;

namespace gtc {
namespace {

inline cudaStream_t as_stream(gtc_stream_t s) { return reinterpret_cast<cudaStream_t>(s); }

// ================================================================ validator

// The reason word starts at kNoReason (every byte 0x7f) so that atomicMin
// keeps the smallest failing reason code; it maps back to GTC_CSR_OK.
constexpr int kNoReason = 0x7f7f7f7f;

// Phase 1: offsets start at 0, end at nnz, never decrease.
template <typename OffT>
__global__ void validate_offsets_kernel(const OffT *__restrict__ off, long long n,
                                        long long nnz, int *reason)
{
    long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v == 0 && ((long long)off[0] != 0 || (long long)off[n] != nnz))
        atomicMin(reason, GTC_CSR_BAD_OFFSETS);
    if (v < n && (long long)off[v + 1] < (long long)off[v])
        atomicMin(reason, GTC_CSR_BAD_OFFSETS);
}

// The row that holds entry e (off[0] <= e < off[n]), found by the whole warp:
// 32 probes cut the range at a time.
template <typename OffT>
__device__ __forceinline__ long long warp_row_of_entry(const OffT *__restrict__ off, long long n,
                                                       long long e)
{
    const int lane = threadIdx.x & 31;
    long long lo = 0, hi = n;                      // off[lo] <= e < off[hi]
    while (hi - lo > 1) {
        const long long step = (hi - lo + 32) / 33;
        const long long at = lo + (lane + 1) * step;
        const unsigned int below = __ballot_sync(0xffffffffu, at < hi && (long long)off[at] <= e);
        const long long k = __popc(below);         // off is non-decreasing: a prefix of the lanes
        hi = min(hi, lo + (k + 1) * step);
        lo += k * step;
    }
    return lo;
}

// A row less than 32 before the one that holds entry e, from row r on (off[r] <=
// e < off[n]): 32 probes at a time, 32 rows apart, then 1,024 and so on while the
// rows have no entries (1 M vertices with 1,000 entries: 4.0 ms in steps of 32
// rows, 0.78 so).
template <typename OffT>
__device__ __forceinline__ long long warp_skip_rows(const OffT *__restrict__ off, long long n,
                                                    long long r, long long e)
{
    const int lane = threadIdx.x & 31;
    for (long long step = 32;;) {
        const long long at = r + (lane + 1) * step;
        const unsigned int below = __ballot_sync(0xffffffffu, at < n && (long long)off[at] <= e);
        const int k = __popc(below);
        r += k * step;
        if (k == 32) step *= 32;
        else if (step > 32) step /= 32;
        else return r;
    }
}

// Phase 2, every entry (a, x) once: x in range, no self-loop, rows strictly
// ascending, and the mirror (x, a) of every entry with a < x present.  If the
// rows are sound, reversal maps the entries with a < x injectively onto those
// with a > x: the graph is symmetric iff every such upper entry's mirror is
// present and both kinds are equally many (counts[0] and counts[1]), so only
// upper entries are searched for, half of all.  The smallest failing reason
// wins, so an unsound row outweighs what its searches say.  Warps take
// kCheckChunk consecutive entries at a time, so that a hub row is spread over
// many; the rows are walked 32 at a time with their ends in the lanes.
constexpr int kCheckChunk = 512;

template <typename OffT>
__global__ void __launch_bounds__(256)
validate_entries_kernel(const OffT *__restrict__ off, const int *__restrict__ ind, long long n,
                        long long nnz, int *reason, unsigned long long *counts)
{
    if (*(volatile int *)reason == GTC_CSR_BAD_OFFSETS) return;
    const int lane = threadIdx.x & 31;
    const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
    unsigned int upper = 0, lower = 0;
    int bad = kNoReason;
    for (long long c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
         c * kCheckChunk < nnz; c += warps) {
        long long e = c * kCheckChunk;
        const long long e1 = min(e + kCheckChunk, nnz);
        long long r = warp_row_of_entry(off, n, e);
        while (e < e1) {
            // lane i: where row r + i ends
            const long long begin = (long long)off[r];
            const long long end = (long long)off[min(r + 1 + lane, n)];
            const long long stop = min(e1, __shfl_sync(0xffffffffu, end, 31));
            if (stop <= e) {
                // 32 rows without entries, maybe of many more
                r = warp_skip_rows(off, n, r + 32, e);
                continue;
            }
            for (; e < stop; e += 32) {
                const long long f = e + lane;
                int i = 0;                         // rows that end at or before f
#pragma unroll
                for (int step = 16; step >= 1; step >>= 1) {
                    const long long at = __shfl_sync(0xffffffffu, end, i + step - 1);
                    if (at <= f) i += step;
                }
                const long long rb = __shfl_sync(0xffffffffu, end, (i - 1) & 31);
                if (f < stop) {
                    const long long a = r + i;
                    const int x = ind[f];
                    const bool in = (unsigned long long)(long long)x < (unsigned long long)n;
                    if (!in) bad = min(bad, (int)GTC_CSR_INDEX_RANGE);
                    else if (x == a) bad = min(bad, (int)GTC_CSR_SELF_LOOP);
                    if (f > (i > 0 ? rb : begin) && ind[f - 1] >= x)
                        bad = min(bad, (int)GTC_CSR_UNSORTED_OR_DUPLICATE);
                    if (x < a) {
                        ++lower;
                    } else {
                        ++upper;
                        if (in) {
                            long long lo = off[x];
                            const long long hi = off[x + 1];
                            int len = (int)(hi - lo);
                            while (len > 0) {
                                const int half = len >> 1;
                                if (ind[lo + half] < a) {
                                    lo += half + 1;
                                    len -= half + 1;
                                } else {
                                    len = half;
                                }
                            }
                            if (lo >= hi || ind[lo] != a)
                                bad = min(bad, (int)GTC_CSR_ASYMMETRIC);
                        }
                    }
                }
            }
            e = stop;
            r = min(r + 32, n - 1);
        }
    }
    bad = __reduce_min_sync(0xffffffffu, bad);
    upper = __reduce_add_sync(0xffffffffu, upper);
    lower = __reduce_add_sync(0xffffffffu, lower);
    if (lane == 0) {
        if (bad != kNoReason) atomicMin(reason, bad);
        if (upper) atomicAdd(&counts[0], (unsigned long long)upper);
        if (lower) atomicAdd(&counts[1], (unsigned long long)lower);
    }
}

template <typename OffT>
gtc_status run_validate(const OffT *off, const int *ind, long long n, long long nnz,
                        void *ws, int32_t *h_reason, cudaStream_t stream)
{
    int *reason = static_cast<int *>(ws);
    unsigned long long *counts =
        reinterpret_cast<unsigned long long *>(static_cast<char *>(ws) + 64);
    cudaError_t e = cudaMemsetAsync(reason, 0x7f, sizeof(int), stream);
    if (e != cudaSuccess) return GTC_ERR_CUDA;
    e = cudaMemsetAsync(counts, 0, 2 * sizeof(unsigned long long), stream);
    if (e != cudaSuccess) return GTC_ERR_CUDA;
    const unsigned vb = (unsigned)div_up<long long>(n + 1, 256);
    validate_offsets_kernel<<<vb, 256, 0, stream>>>(off, n, nnz, reason);
    if (n > 0) {
        int dev = 0, sms = 148;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (nnz > 0) {
            const long long want = div_up<long long>(nnz, 8ll * kCheckChunk);
            const unsigned blocks =
                (unsigned)(want < (long long)sms * 8 ? want : (long long)sms * 8);
            validate_entries_kernel<OffT><<<blocks, 256, 0, stream>>>(off, ind, n, nnz, reason,
                                                                      counts);
        }
    }
    // reason word and the two entry counts in one read
    unsigned char host[80];
    e = cudaMemcpyAsync(host, ws, sizeof(host), cudaMemcpyDeviceToHost, stream);
    if (e != cudaSuccess) return GTC_ERR_CUDA;
    e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return GTC_ERR_CUDA;
    int r = 0;
    unsigned long long c[2] = {0, 0};
    std::memcpy(&r, host, sizeof(int));
    std::memcpy(c, host + 64, sizeof(c));
    if (r == kNoReason && c[0] != c[1]) r = GTC_CSR_ASYMMETRIC;
    *h_reason = r == kNoReason ? GTC_CSR_OK : r;
    return GTC_OK;
}

// ============================================================ vertex subset

constexpr int kSubThreads = 256;
constexpr int kSubWarpRow = 128;                  // longest listed row that a warp takes
constexpr int kSubSlots = 4096;
constexpr long long kSubHubMin = kSubSlots / 2;   // longer listed rows are hubs
constexpr int kSubClaim = 32;                     // most listed vertices that a block takes
constexpr long long kSubFew = 8192;               // of fewer a warp takes half as long rows
constexpr int kSubHubThreads = 1024;
constexpr long long kSubHubBits = 1ll << 20;      // bitmap span of a hub row (128 KiB)

template <typename IndT>
__device__ __forceinline__ bool sorted_contains(const IndT *__restrict__ list,
                                                long long len, long long key)
{
    long long lo = 0, hi = len;
    while (lo < hi) {
        long long mid = (lo + hi) >> 1;
        if ((long long)list[mid] < key) lo = mid + 1; else hi = mid;
    }
    return lo < len && (long long)list[lo] == key;
}

// |N(u) ∩ N(v)| by binary search of the shorter sorted row in the longer,
// this lane's share (lane stride 32).
template <typename IndT>
__device__ __forceinline__ unsigned long long search_shorter(const IndT *__restrict__ ind,
                                                             long long vb, long long dv,
                                                             long long ub, long long du,
                                                             int lane)
{
    unsigned long long acc = 0;
    if (du < dv) {
        for (long long i = lane; i < du; i += 32)
            acc += sorted_contains(ind + vb, dv, (long long)ind[ub + i]);
    } else {
        for (long long i = lane; i < dv; i += 32)
            acc += sorted_contains(ind + ub, du, (long long)ind[vb + i]);
    }
    return acc;
}

__device__ __forceinline__ void add_out(long long *o, unsigned long long x)
{
    atomicAdd(reinterpret_cast<unsigned long long *>(o), x);
}
__device__ __forceinline__ void add_out(int *o, unsigned long long x)
{
    atomicAdd(o, (int)x);
}

// out[k] = sum over u in N(v) of |N(v) ∩ N(u)|, v = vertex[k], with full
// adjacency lists (the rows of the listed vertices and of their neighbours
// are the only ones read, as in the reference's vertex-list kernel,
// src/clusteringCount.cu:266-312).  Edges with u == v or a list shorter
// than two are skipped like the reference (:292-294).  Two kernels:
//   * subset_kernel, rows that are no hubs, a warp for those of at most
//     kSubWarpRow (half of that in lists of less than kSubFew), a block for the
//     others and for every row where the list has no more vertices than there
//     are blocks at a time.  N(v) goes to a shared hash table.  The sum counts
//     adjacent pairs (u, w) of N(v) both ways round, so a pair need be found
//     from one end only: the rows of the short neighbours (not much longer than
//     v's) are looked up in the table, where finding a long w counts twice, and
//     pairs of long neighbours are searched for, one of each two.  It writes 0
//     for the hubs;
//   * subset_hub_kernel, longer ("hub") rows: each block that takes part in a
//     row sets N(v) in a shared bitmap over the row's id span and takes every
//     so-manieth neighbour, whose row its warps probe into the bitmap with
//     coalesced loads; neighbour rows longer than 2,048 entries are queued
//     and swept afterwards by all of the block's warps in 1,024-entry pieces,
//     so that no warp is left alone with a hub's row; block sums are added to
//     out[k].  A row whose span exceeds the bitmap falls back to the binary
//     search.  All blocks take part in a row of more than kSubHubMin: on a
//     power-law graph a single hub's probes outnumber those of thousands of
//     ordinary rows.  Lists of less than 2 kSubFew vertices give it rows from a
//     quarter of that on, too long to be left to one block at the end; those of
//     1,024 vertices are shared out among teams of blocks, down to a block
//     each.  All blocks on one after another take 7 us a row however small it
//     is (2,000 vertices of an ER 100K of mean degree 600: 14.9 ms so, 1.8 by
//     teams, 2.3 with a table and a block each; of 20 cliques of 600, 14.0, 1.15
//     and 0.99 ms).
// A neighbour row is long from here on (elements), for a listed row of dv.
__host__ __device__ __forceinline__ int subset_long(int dv)
{
    return dv > 16 ? 4 * dv : 64;
}

template <typename IndT>
struct SubWarpSmem {
    IndT key[4 * kSubWarpRow];
    unsigned char longs[kSubWarpRow];             // index of each long neighbour in the row
};

template <typename IndT>
struct SubBlockSmem {
    IndT key[kSubSlots];
    unsigned short longs[kSubHubMin];             // index of each long neighbour in the row,
    unsigned short mids[kSubHubMin];              // of each short one of over kSubList entries
};

template <typename IndT>
struct SubSmem {
    union {
        SubWarpSmem<IndT> warp[kSubThreads / 32];
        SubBlockSmem<IndT> block;
    };
    int row[kSubClaim], wide[kSubClaim];          // claimed vertices: warp rows, block rows
    int n_row, n_wide, next, n_long, n_mid;
    unsigned long long sum;
};

template <typename IndT>
__device__ __forceinline__ bool cas_empty(IndT *slot, IndT key)
{
    if (sizeof(IndT) == 4)
        return atomicCAS(reinterpret_cast<int *>(slot), -1, (int)key) == -1;
    return atomicCAS(reinterpret_cast<unsigned long long *>(slot), ~0ull,
                     (unsigned long long)key) == ~0ull;
}

// In N(v)'s table a long neighbour has the top bit set: a byte beside the key
// cost a second shared load per hit.
template <typename IndT>
constexpr IndT kSubFar = (IndT)1 << (8 * sizeof(IndT) - 1);

// What finding w in N(v)'s table counts: 0, 1, or 2 for a long neighbour.
template <typename IndT>
__device__ __forceinline__ unsigned int sub_find(const IndT *key, int lg, IndT w)
{
    const unsigned int mask = (1u << lg) - 1u;
    unsigned int s = hash_slot((int)w, lg);
    IndT k = key[s];
    while ((k & ~kSubFar<IndT>) != w && k != (IndT)-1) {
        s = (s + 1) & mask;
        k = key[s];
    }
    return k == (IndT)-1 ? 0u : (k < 0 ? 2u : 1u);
}

// Neighbour u of v, to the table; true for a long one.  The largest id is never
// taken for one (with the bit it is an empty slot): its row is looked up whole.
template <typename OffT, typename IndT>
__device__ __forceinline__ bool sub_insert(const OffT *__restrict__ off, IndT u, long long v,
                                           int dv, IndT *key, int lg, int &du)
{
    const unsigned int mask = (1u << lg) - 1u;
    const long long d = (long long)off[u + 1] - (long long)off[u];
    const bool lng = u != v && d > subset_long(dv) && u != ~kSubFar<IndT>;
    du = u != v && !lng ? (int)d : 0;
    unsigned int s = hash_slot((int)u, lg);
    while (!cas_empty(&key[s], lng ? (IndT)(u | kSubFar<IndT>) : u)) s = (s + 1) & mask;
    return lng;
}

constexpr int kSubList = 64;                      // longer rows are looked up one by one

// Hits of row u (ub, len) in the table, by the warp, 128 elements at a time; a
// long w counts twice.
template <typename IndT>
__device__ __forceinline__ unsigned int sub_row(const IndT *__restrict__ row, int len,
                                                const IndT *key, int lg)
{
    constexpr int kPer = 4;
    unsigned int acc = 0;
    for (int i0 = threadIdx.x & 31; i0 < len; i0 += 32 * kPer) {
        IndT x[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) x[j] = i0 + 32 * j < len ? row[i0 + 32 * j] : (IndT)-2;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            if (i0 + 32 * j >= len) break;
            acc += sub_find(key, lg, x[j]);
        }
    }
    return acc;
}

// The rows of 32 neighbours of v (this lane's is u, if any) that have at most
// kSubList entries, looked up by the warp as one stream; with `all` also the
// other short ones.
template <typename OffT, typename IndT>
__device__ __forceinline__ unsigned long long
sub_stream(const OffT *__restrict__ off, const IndT *__restrict__ ind, bool has, IndT u,
           long long v, int dv, const IndT *key, int lg, bool all)
{
    constexpr int kPer = 4;
    const int lane = threadIdx.x & 31;
    long long ub = 0;
    int du = 0;
    if (has && u != v) {
        ub = (long long)off[u];
        const long long d = (long long)off[u + 1] - ub;
        du = d >= 2 && (d <= subset_long(dv) || u == ~kSubFar<IndT>) ? (int)d : 0;
    }
    unsigned long long acc = 0;
    unsigned int rows = all ? __ballot_sync(0xffffffffu, du > kSubList) : 0u;
    while (rows) {
        const int src = __ffs(rows) - 1;
        rows &= rows - 1;
        acc += sub_row(ind + __shfl_sync(0xffffffffu, ub, src),
                       __shfl_sync(0xffffffffu, du, src), key, lg);
    }
    const int len = du <= kSubList ? du : 0;
    const int incl = warp_incl_scan(len);
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    const long long start = ub - (incl - len);
    for (int f0 = 0; f0 < total; f0 += 32 * kPer) {
        IndT x[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int f = f0 + 32 * j + lane;
            const long long at = __shfl_sync(0xffffffffu, start, warp_corank(incl, f));
            x[j] = f < total ? ind[at + f] : (IndT)-2;
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            acc += sub_find(key, lg, x[j]);
        }
    }
    return acc;
}

// Pairs first, first + stride, ... of the n long neighbours longs[] of v:
// whether the one is in the other's row, the shorter of the two.
template <typename OffT, typename IndT, typename Idx>
__device__ __forceinline__ unsigned long long
sub_pairs(const OffT *__restrict__ off, const IndT *__restrict__ ind, long long vb,
          const Idx *longs, int n, int first, int stride)
{
    constexpr int kPer = 4;                        // searches in flight per thread
    const int pairs = n * (n - 1) / 2;
    unsigned long long acc = 0;
    for (int p0 = first; p0 < pairs; p0 += kPer * stride) {
        IndT key[kPer];
        long long lo[kPer];
        long long len[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int p = p0 + j * stride;
            len[j] = 0;
            if (p >= pairs) continue;
            int i = (int)((sqrtf(8.0f * (float)p + 1.0f) + 1.0f) * 0.5f);
            while (i * (i - 1) / 2 > p) --i;
            while (i * (i + 1) / 2 <= p) ++i;
            const IndT a = ind[vb + longs[i]], b = ind[vb + longs[p - i * (i - 1) / 2]];
            const long long ab = off[a], da = (long long)off[a + 1] - ab;
            const long long bb = off[b], db = (long long)off[b + 1] - bb;
            lo[j] = da < db ? ab : bb;
            len[j] = da < db ? da : db;
            key[j] = da < db ? b : a;
        }
        bool more = true;
        while (more) {
            IndT x[kPer];
#pragma unroll
            for (int j = 0; j < kPer; ++j)
                x[j] = len[j] > 0 ? ind[lo[j] + (len[j] >> 1)] : (IndT)-1;
            more = false;
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                if (len[j] <= 0) continue;
                const long long half = len[j] >> 1;
                if (x[j] < key[j]) {
                    lo[j] += half + 1;
                    len[j] -= half + 1;
                } else {
                    acc += x[j] == key[j];
                    len[j] = x[j] == key[j] ? 0 : half;
                }
                more |= len[j] > 0;
            }
        }
    }
    return 2 * acc;
}

template <typename OffT, typename IndT, typename VtxT, typename OutT>
__global__ void __launch_bounds__(kSubThreads, 4)
subset_kernel(const OffT *__restrict__ off, const IndT *__restrict__ ind,
              const VtxT *__restrict__ vertex, long long count, OutT *__restrict__ out,
              const int *__restrict__ skip, int claim, int warp_row, int hub_min)
{
    extern __shared__ __align__(16) unsigned char smem[];
    SubSmem<IndT> &sm = *reinterpret_cast<SubSmem<IndT> *>(smem);
    if (skip && *skip) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // a row by the whole block
    auto block_row = [&](long long k, long long v, long long vb, int dv) {
        const int lg = ceil_log2(dv > 16 ? 2 * (long long)dv : 32);
        __syncthreads();
        if (threadIdx.x == 0) { sm.sum = 0; sm.n_long = sm.n_mid = sm.next = 0; }
        for (int i = threadIdx.x; i < (1 << lg); i += kSubThreads) sm.block.key[i] = (IndT)-1;
        __syncthreads();
        for (int i = threadIdx.x; i < dv; i += kSubThreads) {
            int du;
            if (sub_insert(off, ind[vb + i], v, dv, sm.block.key, lg, du))
                sm.block.longs[atomicAdd(&sm.n_long, 1)] = (unsigned short)i;
            else if (du > kSubList)
                sm.block.mids[atomicAdd(&sm.n_mid, 1)] = (unsigned short)i;
        }
        __syncthreads();
        unsigned long long acc = 0;
        // the lanes find where 32 neighbours' rows are, which the warp then takes in turn
        constexpr int kWarps = kSubThreads / 32;
        for (int i0 = warp; i0 < sm.n_mid; i0 += 32 * kWarps) {
            long long ub = 0;
            int du = 0;
            if (i0 + kWarps * lane < sm.n_mid) {
                const IndT u = ind[vb + sm.block.mids[i0 + kWarps * lane]];
                ub = off[u];
                du = (int)((long long)off[u + 1] - ub);
            }
            const int n = min(32, div_up(sm.n_mid - i0, kWarps));
            for (int k = 0; k < n; ++k)
                acc += sub_row(ind + __shfl_sync(0xffffffffu, ub, k),
                               __shfl_sync(0xffffffffu, du, k), sm.block.key, lg);
        }
        // a share of the neighbours that keeps all warps busy on a short row
        const int each = min(32, max(4, div_up(dv, kWarps)));
        const int from = sm.n_mid + sm.n_long < dv ? warp * each : dv;    // none left
        for (int i = from; i < dv; i += each * kWarps) {
            const bool has = lane < each && i + lane < dv;
            acc += sub_stream(off, ind, has, has ? ind[vb + i + lane] : (IndT)0, v, dv,
                              sm.block.key, lg, false);
        }
        acc += sub_pairs(off, ind, vb, sm.block.longs, sm.n_long, (int)threadIdx.x,
                         kSubThreads);
        const unsigned long long ws =
            cg::reduce(cg::tiled_partition<32>(cg::this_thread_block()), acc,
                       cg::plus<unsigned long long>());
        if (lane == 0 && ws) atomicAdd(&sm.sum, ws);
        __syncthreads();
        if (threadIdx.x == 0) { out[k] = (OutT)sm.sum; sm.next = 0; }
    };
    if (claim == 1) {
        for (long long k = blockIdx.x; k < count; k += gridDim.x) {
            const long long v = (long long)vertex[k];
            const long long vb = off[v], dv = (long long)off[v + 1] - vb;
            if (dv < 2 || dv > hub_min) {
                if (threadIdx.x == 0) out[k] = 0;
            } else {
                block_row(k, v, vb, (int)dv);
            }
        }
        return;
    }
    const long long claims = div_up<long long>(count, claim);
    for (long long c = blockIdx.x; c < claims; c += gridDim.x) {
        // part the claimed vertices (spread over the list) by row length
        __syncthreads();
        if (threadIdx.x < 32) {
            const long long k = c + claims * threadIdx.x;
            long long dv = -1;
            if (lane < claim && k < count) {
                const long long v = (long long)vertex[k];
                dv = (long long)off[v + 1] - (long long)off[v];
                if (dv > hub_min) out[k] = 0;
            }
            const unsigned int below = (1u << lane) - 1u;
            const bool narrow = dv >= 0 && dv <= warp_row;
            const bool wide = dv > warp_row && dv <= hub_min;
            const unsigned int mn = __ballot_sync(0xffffffffu, narrow);
            const unsigned int mw = __ballot_sync(0xffffffffu, wide);
            if (narrow) sm.row[__popc(mn & below)] = lane;
            if (wide) sm.wide[__popc(mw & below)] = lane;
            if (lane == 0) {
                sm.n_row = __popc(mn);
                sm.n_wide = __popc(mw);
                sm.next = 0;
            }
        }
        __syncthreads();
        for (int r = 0; r < sm.n_wide; ++r) {
            const long long k = c + claims * sm.wide[r];
            const long long v = (long long)vertex[k];
            block_row(k, v, off[v], (int)((long long)off[v + 1] - (long long)off[v]));
        }
        __syncthreads();
        SubWarpSmem<IndT> &ws = sm.warp[warp];
        while (true) {
            int r = 0;
            if (lane == 0) r = atomicAdd(&sm.next, 1);
            r = __shfl_sync(0xffffffffu, r, 0);
            if (r >= sm.n_row) break;
            const long long k = c + claims * sm.row[r];
            const long long v = (long long)vertex[k];
            const long long vb = off[v];
            const int dv = (int)((long long)off[v + 1] - vb);
            const int lg = ceil_log2(dv > 8 ? 4 * (long long)dv : 32);
            __syncwarp();
            for (int i = lane; i < (1 << lg); i += 32) ws.key[i] = (IndT)-1;
            __syncwarp();
            int n_long = 0;
            for (int i0 = 0; i0 < dv; i0 += 32) {
                const bool has = i0 + lane < dv;
                int du;
                const bool lng =
                    has && sub_insert(off, ind[vb + i0 + lane], v, dv, ws.key, lg, du);
                const unsigned int m = __ballot_sync(0xffffffffu, lng);
                if (lng) ws.longs[n_long + __popc(m & ((1u << lane) - 1u))] =
                    (unsigned char)(i0 + lane);
                n_long += __popc(m);
            }
            __syncwarp();
            unsigned long long acc = 0;
            if (dv >= 2) {
                for (int i0 = 0; i0 < dv; i0 += 32) {
                    const bool has = i0 + lane < dv;
                    acc += sub_stream(off, ind, has, has ? ind[vb + i0 + lane] : (IndT)0, v, dv,
                                      ws.key, lg, true);
                }
                acc += sub_pairs(off, ind, vb, ws.longs, n_long, lane, 32);
            }
            acc = cg::reduce(cg::tiled_partition<32>(cg::this_thread_block()), acc,
                             cg::plus<unsigned long long>());
            if (lane == 0) out[k] = (OutT)acc;
        }
    }
}

// What the listed vertices' own rows cost, in looked-up elements (a search in
// a long row as 16), against counting the whole graph: *whole is set when they
// are more than kSubWhole per adjacency entry, or when one row that a block
// takes alone is more than one per kSubRow entries.  R-MAT graphs count at some
// 50 ps an entry (uniform ones at half of that); listed rows take some 5 ps an
// element, 1 ns for a block alone.
constexpr unsigned long long kSubWhole = 16, kSubRow = 16;

template <typename OffT>
__global__ void subset_cost_kernel(const OffT *__restrict__ off, const int *__restrict__ ind,
                                   const int *__restrict__ vertex, long long count,
                                   unsigned long long limit, unsigned long long *cost, int *whole)
{
    const int lane = threadIdx.x & 31;
    const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
    unsigned long long mine = 0;
    for (long long k = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < count;
         k += warps) {
        const long long v = vertex[k], vb = off[v];
        const int dv = (int)((long long)off[v + 1] - vb);
        const bool hub = dv > kSubHubMin;
        // 128 neighbours at a time; of a longer row than 256, a sample
        const int each = dv > 256 ? dv / 256 : 1;
        unsigned int longs = 0;
        for (int i0 = 0; i0 < dv; i0 += 128 * each) {
            long long du[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int i = i0 + 32 * j + lane;
                const int u = i < dv ? ind[vb + i] : -1;
                du[j] = u >= 0 ? (long long)off[u + 1] - (long long)off[u] : -1;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (du[j] < 0) continue;
                if (hub || du[j] <= subset_long(dv)) mine += (unsigned long long)du[j] * each;
                else longs += each;
            }
        }
        longs = __reduce_add_sync(0xffffffffu, longs);
        const unsigned long long pairs = 8ull * longs * longs;
        if (lane == 0) {
            mine += pairs;
            if (!hub && pairs * kSubRow > limit / kSubWhole) *whole = 1;
        }
    }
    mine = cg::reduce(cg::tiled_partition<32>(cg::this_thread_block()), mine,
                      cg::plus<unsigned long long>());
    if (lane == 0 && mine) {
        const unsigned long long before = atomicAdd(cost, mine);
        if (before <= limit && before + mine > limit) *whole = 1;
    }
}

// r of the listed vertices after a count of the whole graph (*whole set).
__global__ void subset_gather_kernel(const Data w, const int *__restrict__ vertex,
                                     long long count, long long *__restrict__ out)
{
    if (!*w.gate) return;
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const int v = vertex[k];
    unsigned long long t = w.tacc[v];
    const int key = w.key[v];
    if (key > kKeyTop - w.recs[0].core) t += w.tcore[kKeyTop - key];
    out[k] = (long long)(2 * t);
}

template <typename OffT, typename IndT, typename VtxT, typename OutT>
__global__ void __launch_bounds__(kSubHubThreads, 1)
subset_hub_kernel(const OffT *__restrict__ off, const IndT *__restrict__ ind,
                      const VtxT *__restrict__ vertex, long long count,
                  OutT *__restrict__ out, const int *__restrict__ skip, long long hub_min)
{
    extern __shared__ unsigned int s_bits[];          // kSubHubBits / 32 words
    if (skip && *skip) return;
    // all blocks' rows from the front, teams' from the end
    __shared__ long long s_hub[kSubHubThreads];
    __shared__ int s_all[kSubHubThreads / 32], s_team[kSubHubThreads / 32];
    __shared__ long long s_lo, s_hi;
    __shared__ unsigned long long s_sum;
    constexpr int kBigRows = 64, kSplit = 2048, kPiece = 1024;
    __shared__ long long s_big_b[kBigRows], s_big_e[kBigRows];
    __shared__ int s_nbig;
    auto block = cg::this_thread_block();
    auto warp = cg::tiled_partition<32>(block);
    const int wid = warp.meta_group_rank(), lane = warp.thread_rank();
    constexpr int nwarps = kSubHubThreads / 32;
    // the listed vertices are scanned a chunk at a time, every thread testing
    // one; all blocks find the same rows in the same order
    for (long long c0 = 0; c0 < count; c0 += kSubHubThreads) {
        const long long kk = c0 + threadIdx.x;
        long long dk = 0;
        if (kk < count) {
            const long long v = (long long)vertex[kk];
            dk = (long long)off[v + 1] - (long long)off[v];
        }
        if (!__syncthreads_or(dk > hub_min)) continue;
        const bool all = dk > kSubHubMin, team = !all && dk > hub_min;
        const unsigned int ma = __ballot_sync(0xffffffffu, all);
        const unsigned int mt = __ballot_sync(0xffffffffu, team);
        if (lane == 0) {
            s_all[wid] = __popc(ma);
            s_team[wid] = __popc(mt);
        }
        __syncthreads();
        int na = 0, nt = 0, a0 = 0, t0 = 0;
        for (int i = 0; i < nwarps; ++i) {
            if (i == wid) {
                a0 = na;
                t0 = nt;
            }
            na += s_all[i];
            nt += s_team[i];
        }
        const unsigned int below = (1u << lane) - 1u;
        if (all) s_hub[a0 + __popc(ma & below)] = kk;
        if (team) s_hub[kSubHubThreads - 1 - (t0 + __popc(mt & below))] = kk;
        __syncthreads();
        // rows for teams: as many teams of blocks as there are rows, if there are enough blocks
        const int blocks = nt > 0 ? max(1, (int)gridDim.x / nt) : 1;
        const int teams = (int)gridDim.x / blocks;
        const int mine = (int)blockIdx.x / blocks;
        const int rows = mine < teams && mine < nt ? div_up(nt - mine, teams) : 0;
        for (int h = 0; h < na + rows; ++h) {
            const bool whole = h < na;
            const long long k = s_hub[whole ? h : kSubHubThreads - 1 - (mine + (h - na) * teams)];
            const int size = whole ? (int)gridDim.x : blocks;
            const int rank = whole ? (int)blockIdx.x : (int)blockIdx.x % blocks;
            const long long stride = (long long)size * nwarps;    // neighbours per step
            const long long v = (long long)vertex[k];
            const long long vb = off[v], ve = off[v + 1], dv = ve - vb;
            // the row's id span (rows are sorted, but the bitmap must not
            // depend on it)
            long long lo = LLONG_MAX, hi = LLONG_MIN;
            for (long long i = vb + threadIdx.x; i < ve; i += kSubHubThreads) {
                const long long x = (long long)ind[i];
                lo = min(lo, x);
                hi = max(hi, x);
            }
            lo = cg::reduce(warp, lo, cg::less<long long>());
            hi = cg::reduce(warp, hi, cg::greater<long long>());
            if (threadIdx.x == 0) { s_lo = LLONG_MAX; s_hi = LLONG_MIN; s_sum = 0; s_nbig = 0; }
            __syncthreads();
            if (lane == 0) { atomicMin(&s_lo, lo); atomicMax(&s_hi, hi); }
            __syncthreads();
            lo = s_lo;
            hi = s_hi;
            const unsigned long long span = (unsigned long long)(hi - lo) + 1ull;
            const bool use_bits = span <= (unsigned long long)kSubHubBits;
            if (use_bits) {
                const int words = (int)((span + 31) >> 5);
                for (int i = threadIdx.x; i < words; i += kSubHubThreads) s_bits[i] = 0;
                __syncthreads();
                for (long long i = vb + threadIdx.x; i < ve; i += kSubHubThreads) {
                    const unsigned long long x = (unsigned long long)((long long)ind[i] - lo);
                    atomicOr(&s_bits[x >> 5], 1u << (x & 31));
                }
                __syncthreads();
            }
            unsigned long long acc = 0;
            typedef typename std::make_unsigned<IndT>::type Id;
            const Id first = (Id)lo, last = use_bits ? (Id)span : 0;
            auto sweep = [&](long long b0, long long b1) {
                constexpr int kPer = 32 / sizeof(IndT);    // loads in flight per lane
                for (long long i0 = b0 + lane; i0 < b1; i0 += 32 * kPer) {
                    Id x[kPer];
#pragma unroll
                    for (int j = 0; j < kPer; ++j)
                        x[j] = i0 + 32 * j < b1 ? (Id)ind[i0 + 32 * j] - first : last;
                    unsigned int hits = 0;
#pragma unroll
                    for (int j = 0; j < kPer; ++j)
                        if (x[j] < last) hits += (s_bits[x[j] >> 5] >> (x[j] & 31)) & 1u;
                    acc += hits;
                }
            };
            // the lanes find where 32 neighbours' rows are, which the warp then takes in turn
            for (long long e0 = vb + rank + (long long)size * wid; e0 < ve; e0 += 32 * stride) {
                long long ub = 0, ue = 0;
                if (e0 + lane * stride < ve) {
                    const long long u = (long long)ind[e0 + lane * stride];
                    ub = off[u];
                    ue = u == v ? ub : (long long)off[u + 1];
                }
                unsigned int todo = __ballot_sync(0xffffffffu, ue - ub >= 2);
                while (todo) {
                    const int src = __ffs(todo) - 1;
                    todo &= todo - 1;
                    const long long b0 = __shfl_sync(0xffffffffu, ub, src);
                    const long long b1 = __shfl_sync(0xffffffffu, ue, src);
                    if (use_bits && b1 - b0 > kSplit) {
                        // a long row is shared by the block's warps after this loop
                        int at = 0;
                        if (lane == 0) at = atomicAdd(&s_nbig, 1);
                        at = warp.shfl(at, 0);
                        if (at < kBigRows) {
                            if (lane == 0) { s_big_b[at] = b0; s_big_e[at] = b1; }
                            continue;
                        }
                    }
                    if (use_bits) sweep(b0, b1);
                    else acc += search_shorter(ind, vb, dv, b0, b1 - b0, lane);
                }
            }
            if (use_bits) {
                __syncthreads();
                const int nbig = min(s_nbig, kBigRows);
                for (int r = 0; r < nbig; ++r) {
                    const long long b0 = s_big_b[r], b1 = s_big_e[r];
                    for (long long c0 = b0 + (long long)wid * kPiece; c0 < b1;
                         c0 += (long long)nwarps * kPiece)
                        sweep(c0, c0 + kPiece < b1 ? c0 + kPiece : b1);
                }
            }
            const unsigned long long ws = cg::reduce(warp, acc, cg::plus<unsigned long long>());
            if (lane == 0 && ws) atomicAdd(&s_sum, ws);
            __syncthreads();
            if (threadIdx.x == 0 && s_sum) add_out(&out[k], s_sum);
            __syncthreads();                       // s_bits, s_lo and s_sum are reused
        }
    }
}

// skip: device flag (nullable); set, the kernels leave out as it is.
template <typename OffT, typename IndT, typename VtxT, typename OutT>
gtc_status launch_subset(const OffT *off, const IndT *ind, const VtxT *vertex,
                         long long count, OutT *out, cudaStream_t stream,
                         const int *skip = nullptr)
{
    if (count <= 0) return GTC_OK;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    auto rows = subset_kernel<OffT, IndT, VtxT, OutT>;
    constexpr int rsmem = (int)sizeof(SubSmem<IndT>);
    static_assert(rsmem <= 48 * 1024, "what a launch may have without asking");
    // the vertices in as many shares as there are blocks at a time, or whole
    // multiples of that, up to kSubClaim a share: 60,000 vertices of an ER 100K of
    // mean degree 600 take 74 ms so, 98 at 32 a share and 1,184 blocks that took
    // one share after another; rows of R-MAT 18 6.3 and 6.4 ms
    const bool few = count < kSubFew;
    const long long fit = 4ll * sms;
    const int claim = (int)div_up(count, fit * div_up(count, fit * kSubClaim));
    const long long hub_min = count < 2 * kSubFew ? kSubHubMin / 4 : kSubHubMin;
    const long long claims = div_up<long long>(count, claim);
    const long long blocks = min(claims, (long long)INT_MAX);
    rows<<<(unsigned)blocks, kSubThreads, rsmem, stream>>>(
        off, ind, vertex, count, out, skip, claim, few ? kSubWarpRow / 2 : kSubWarpRow, (int)hub_min);
    // the hub kernel adds to what subset_kernel wrote (0 for hubs), in
    // stream order
    auto hub = subset_hub_kernel<OffT, IndT, VtxT, OutT>;
    const int smem = (int)(kSubHubBits / 8);
    if (cudaFuncSetAttribute(hub, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
        cudaSuccess)
        return GTC_ERR_CUDA;
    hub<<<(unsigned)sms, kSubHubThreads, smem, stream>>>(off, ind, vertex, count, out, skip, hub_min);
    return cudaGetLastError() == cudaSuccess ? GTC_OK : GTC_ERR_CUDA;
}

// Whether counting the whole graph may be the cheaper way to a subset of
// `count` of its n vertices: on R-MAT graphs it is from some n / 200 on.  The
// estimate and the launches that end at once cost 35 us, which fewer vertices
// of a uniform graph take altogether.
bool subset_may_count(long long n, long long nnz, long long count)
{
    return nnz > 0 && count >= 16384 && n <= 256 * count;
}

// A subset of a graph of known size, with a workspace: a cost estimate on the
// device picks between the listed rows and a count of the whole graph, whose
// kernels end at once when they are not picked.
template <typename OffT>
gtc_status launch_subset_ws(const OffT *off, const int *ind, long long n, long long nnz,
                            const int *vertex, long long count, long long *out, void *ws,
                            size_t ws_bytes, cudaStream_t stream)
{
    unsigned long long *cost = static_cast<unsigned long long *>(ws);
    int *whole = reinterpret_cast<int *>(cost + 1);
    if (cudaMemsetAsync(ws, 0, 16, stream) != cudaSuccess) return GTC_ERR_CUDA;
    const long long want = div_up<long long>(count, 8);
    subset_cost_kernel<OffT><<<(unsigned)(want < 1184 ? want : 1184), 256, 0, stream>>>(
        off, ind, vertex, count, kSubWhole * (unsigned long long)nnz, cost, whole);
    Data w;
    RowConfig cfg = pick_row_config(n, nnz);
    cfg.split = false;
    gtc_status st = run_count<OffT>(off, ind, n, nnz, true, nullptr, nullptr, nullptr, nullptr,
                                    static_cast<char *>(ws) + 256, ws_bytes - 256, stream,
                                    cfg, nullptr, nullptr, whole, &w);
    if (st != GTC_OK) return st;
    subset_gather_kernel<<<(unsigned)div_up<long long>(count, 256), 256, 0, stream>>>(w, vertex,
                                                                                     count, out);
    return launch_subset(off, ind, vertex, count, out, stream, whole);
}

// ================================================================== compat

// int64 neighbour ids -> int32.  An id outside [0, nv) becomes -1, which the
// counting kernels flag (kErrIndexRange) and skip, so a wide id can never
// wrap into a valid-looking one.
__global__ void narrow_kernel(const long long *__restrict__ in, int *__restrict__ out,
                              long long count, long long nv)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) {
        const long long x = in[i];
        out[i] = (x >= 0 && x < nv) ? (int)x : -1;
    }
}

__global__ void narrow_out_kernel(const long long *__restrict__ in, int *__restrict__ out,
                                  long long count)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) out[i] = (int)in[i];
}

struct CompatCache {
    void *ptr = nullptr;
    size_t bytes = 0;
};
std::mutex g_compat_mu;
CompatCache g_compat[64];
thread_local gtc_status g_compat_status = GTC_OK;
// Workspace of this thread's last kernelCall shim that launched a count
// (its status word is read by gtc_compat_last_status), or null.
thread_local const void *g_compat_ws = nullptr;

// Device error bits -> status.
gtc_status status_from_bits(unsigned int bits)
{
    return (bits & kErrIndexRange) ? GTC_ERR_INVALID_CSR : GTC_OK;
}

void *compat_workspace(size_t bytes)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lock(g_compat_mu);
    CompatCache &c = g_compat[dev];
    if (c.bytes < bytes) {
        if (c.ptr) cudaFree(c.ptr);
        c.ptr = nullptr;
        c.bytes = 0;
        if (cudaMalloc(&c.ptr, bytes) != cudaSuccess) { c.ptr = nullptr; return nullptr; }
        c.bytes = bytes;
    }
    return c.ptr;
}

bool compat_block_size_ok(unsigned int bs)
{
    switch (bs) {
    case 32: case 64: case 96: case 128: case 192: case 256: case 512: case 1024: return true;
    default: return false;
    }
}

}  // namespace
}  // namespace gtc

using namespace gtc;

extern "C" {

const char *gtc_status_string(gtc_status s)
{
    switch (s) {
    case GTC_OK: return "ok";
    case GTC_ERR_INVALID_ARGUMENT: return "invalid argument";
    case GTC_ERR_INVALID_CSR: return "invalid CSR";
    case GTC_ERR_WORKSPACE_TOO_SMALL: return "workspace too small";
    case GTC_ERR_CUDA: return "CUDA runtime error";
    case GTC_ERR_OUT_OF_MEMORY: return "out of device memory";
    case GTC_ERR_UNSUPPORTED: return "unsupported device or configuration";
    case GTC_ERR_TIMEOUT: return "bounded device wait timed out";
    case GTC_ERR_CAPACITY: return "capacity exceeded";
    case GTC_ERR_BUSY: return "busy";
    }
    return "unknown status";
}

gtc_status gtc_device_info(int *sm_count, int *cc)
{
    if (!sm_count || !cc) return GTC_ERR_INVALID_ARGUMENT;
    int dev = 0, major = 0, minor = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return GTC_ERR_CUDA;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev) != cudaSuccess)
        return GTC_ERR_CUDA;
    *sm_count = sms;
    *cc = major * 10 + minor;
    return GTC_OK;
}

gtc_status gtc_workspace_size(int64_t n, int64_t nnz, int off_bits, gtc_mode mode, size_t *bytes)
{
    if (!bytes || n < 0 || nnz < 0 || (off_bits != 32 && off_bits != 64)) return GTC_ERR_INVALID_ARGUMENT;
    if (mode != GTC_MODE_PLAIN && mode != GTC_MODE_ORIENTED) return GTC_ERR_INVALID_ARGUMENT;
    if (n > 0x7fffffffll) return GTC_ERR_UNSUPPORTED;           // int32 vertex ids
    if (off_bits == 32 && nnz > 0x7fffffffll) return GTC_ERR_INVALID_ARGUMENT;
    *bytes = make_plan(n, nnz, off_bits, mode == GTC_MODE_PLAIN).bytes;
    return GTC_OK;
}

gtc_status gtc_count_launches(int64_t n, int64_t nnz, gtc_mode mode,
                              const gtc_tuning *tuning, int *launches, int *labels)
{
    if (n < 0 || nnz < 0 || !launches || !labels ||
        (mode != GTC_MODE_PLAIN && mode != GTC_MODE_ORIENTED))
        return GTC_ERR_INVALID_ARGUMENT;
    RowConfig cfg = pick_row_config(n, nnz);
    const gtc_status st = apply_tuning(cfg, tuning);
    if (st != GTC_OK) return st;
    *launches = launches_per_count(cfg, mode == GTC_MODE_PLAIN, n);
    *labels = cfg.split ? GTC_LABELS_DEGREE_RANK : GTC_LABELS_VERTEX_ID;
    return GTC_OK;
}

gtc_status gtc_count_tuned(const void *d_off, int off_bits, const int32_t *d_ind, int64_t n,
                           int64_t nnz, gtc_mode mode, int64_t *d_r, int64_t *d_t,
                           double *d_lcc, int64_t *d_global, void *d_workspace, size_t ws_bytes,
                           gtc_stream_t stream, const gtc_tuning *tuning)
{
    size_t need = 0;
    gtc_status st = gtc_workspace_size(n, nnz, off_bits, mode, &need);
    if (st != GTC_OK) return st;
    if (!d_off || (nnz > 0 && !d_ind) || !d_workspace) return GTC_ERR_INVALID_ARGUMENT;
    if (mode == GTC_MODE_ORIENTED && (d_r || d_t || d_lcc)) return GTC_ERR_INVALID_ARGUMENT;
    if (reinterpret_cast<uintptr_t>(d_workspace) & 255) return GTC_ERR_INVALID_ARGUMENT;
    const bool pv = mode == GTC_MODE_PLAIN;
    if (ws_bytes < make_plan(n, nnz, off_bits, pv).need) return GTC_ERR_WORKSPACE_TOO_SMALL;
    RowConfig cfg = pick_row_config(n, nnz);
    st = apply_tuning(cfg, tuning);
    if (st != GTC_OK) return st;
    long long *r = reinterpret_cast<long long *>(d_r);
    long long *t = reinterpret_cast<long long *>(d_t);
    long long *g = reinterpret_cast<long long *>(d_global);
    if (off_bits == 32)
        return run_count<int>(static_cast<const int *>(d_off), d_ind, n, nnz, pv, r, t, d_lcc, g,
                              d_workspace, ws_bytes, as_stream(stream), cfg, nullptr);
    return run_count<long long>(static_cast<const long long *>(d_off), d_ind, n, nnz, pv, r, t,
                                d_lcc, g, d_workspace, ws_bytes, as_stream(stream), cfg, nullptr);
}

gtc_status gtc_count(const void *d_off, int off_bits, const int32_t *d_ind, int64_t n,
                     int64_t nnz, gtc_mode mode, int64_t *d_r, int64_t *d_t, double *d_lcc,
                     int64_t *d_global, void *d_workspace, size_t ws_bytes, gtc_stream_t stream)
{
    return gtc_count_tuned(d_off, off_bits, d_ind, n, nnz, mode, d_r, d_t, d_lcc, d_global,
                           d_workspace, ws_bytes, stream, nullptr);
}

gtc_status gtc_count_phase_times(const void *d_off, int off_bits, const int32_t *d_ind,
                                 int64_t n, int64_t nnz, void *d_workspace, size_t ws_bytes,
                                 float *h_ms, const gtc_tuning *tuning)
{
    size_t need = 0;
    gtc_status st = gtc_workspace_size(n, nnz, off_bits, GTC_MODE_PLAIN, &need);
    if (st != GTC_OK) return st;
    if (!d_off || (nnz > 0 && !d_ind) || !d_workspace || !h_ms) return GTC_ERR_INVALID_ARGUMENT;
    if (ws_bytes < make_plan(n, nnz, off_bits, true).need) return GTC_ERR_WORKSPACE_TOO_SMALL;
    RowConfig cfg = pick_row_config(n, nnz);
    st = apply_tuning(cfg, tuning);
    if (st != GTC_OK) return st;
    CountTimings tm;
    for (int i = 0; i < 5; ++i)
        if (cudaEventCreate(&tm.ev[i]) != cudaSuccess) return GTC_ERR_CUDA;
    if (off_bits == 32)
        st = run_count<int>(static_cast<const int *>(d_off), d_ind, n, nnz, true, nullptr,
                            nullptr, nullptr, nullptr, d_workspace, ws_bytes, 0, cfg, &tm);
    else
        st = run_count<long long>(static_cast<const long long *>(d_off), d_ind, n, nnz, true,
                                  nullptr, nullptr, nullptr, nullptr, d_workspace, ws_bytes, 0,
                                  cfg, &tm);
    if (st == GTC_OK && cudaEventSynchronize(tm.ev[4]) != cudaSuccess) st = GTC_ERR_CUDA;
    if (st == GTC_OK && n > 0) {
        for (int i = 0; i < 4; ++i) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, tm.ev[i], tm.ev[i + 1]);
            h_ms[i] = ms;
        }
    }
    for (int i = 0; i < 5; ++i) cudaEventDestroy(tm.ev[i]);
    return st;
}

size_t gtc_validate_workspace_size(int64_t n, int64_t nnz)
{
    (void)n;
    (void)nnz;
    return 256;
}

gtc_status gtc_validate_csr(const void *d_off, int off_bits, const int32_t *d_ind, int64_t n,
                            int64_t nnz, void *d_workspace, size_t ws_bytes, int32_t *h_reason,
                            gtc_stream_t stream)
{
    if (!d_off || (nnz > 0 && !d_ind) || !d_workspace || !h_reason || n < 0 || nnz < 0)
        return GTC_ERR_INVALID_ARGUMENT;
    if (off_bits != 32 && off_bits != 64) return GTC_ERR_INVALID_ARGUMENT;
    if (n > 0x7fffffffll) return GTC_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(d_workspace) & 255) return GTC_ERR_INVALID_ARGUMENT;
    if (ws_bytes < gtc_validate_workspace_size(n, nnz)) return GTC_ERR_WORKSPACE_TOO_SMALL;
    if (off_bits == 32)
        return run_validate<int>(static_cast<const int *>(d_off), d_ind, n, nnz, d_workspace,
                                 h_reason, as_stream(stream));
    return run_validate<long long>(static_cast<const long long *>(d_off), d_ind, n, nnz,
                                   d_workspace, h_reason, as_stream(stream));
}

gtc_status gtc_count_subset(const void *d_off, int off_bits, const int32_t *d_ind,
                            const int32_t *d_vertex, int64_t count, int64_t *d_out,
                            gtc_stream_t stream)
{
    if (count < 0) return GTC_ERR_INVALID_ARGUMENT;
    if (count == 0) return GTC_OK;
    if (!d_off || !d_ind || !d_vertex || !d_out) return GTC_ERR_INVALID_ARGUMENT;
    if (off_bits == 32)
        return launch_subset(static_cast<const int *>(d_off), d_ind, d_vertex, count,
                             reinterpret_cast<long long *>(d_out), as_stream(stream));
    if (off_bits == 64)
        return launch_subset(static_cast<const long long *>(d_off), d_ind, d_vertex, count,
                             reinterpret_cast<long long *>(d_out), as_stream(stream));
    return GTC_ERR_INVALID_ARGUMENT;
}

gtc_status gtc_subset_workspace_size(int64_t n, int64_t nnz, int off_bits, int64_t count,
                                     size_t *bytes)
{
    if (!bytes || n < 0 || nnz < 0 || count < 0 || (off_bits != 32 && off_bits != 64))
        return GTC_ERR_INVALID_ARGUMENT;
    *bytes = 0;
    if (n <= 0x7fffffffll && subset_may_count(n, nnz, count))
        *bytes = 256 + make_plan(n, nnz, off_bits, true).bytes;
    return GTC_OK;
}

gtc_status gtc_count_subset_ws(const void *d_off, int off_bits, const int32_t *d_ind, int64_t n,
                               int64_t nnz, const int32_t *d_vertex, int64_t count,
                               int64_t *d_out, void *d_workspace, size_t ws_bytes,
                               gtc_stream_t stream)
{
    size_t need = 0;
    const gtc_status st = gtc_subset_workspace_size(n, nnz, off_bits, count, &need);
    if (st != GTC_OK) return st;
    if (need == 0 || ws_bytes < 256 + make_plan(n, nnz, off_bits, true).need)
        return gtc_count_subset(d_off, off_bits, d_ind, d_vertex, count, d_out, stream);
    if (!d_off || !d_ind || !d_vertex || !d_out || !d_workspace ||
        (reinterpret_cast<uintptr_t>(d_workspace) & 255))
        return GTC_ERR_INVALID_ARGUMENT;
    long long *out = reinterpret_cast<long long *>(d_out);
    if (off_bits == 32)
        return launch_subset_ws(static_cast<const int *>(d_off), d_ind, n, nnz, d_vertex, count,
                                out, d_workspace, ws_bytes, as_stream(stream));
    return launch_subset_ws(static_cast<const long long *>(d_off), d_ind, n, nnz, d_vertex, count,
                            out, d_workspace, ws_bytes, as_stream(stream));
}

gtc_status gtc_compat_last_status(void)
{
    if (g_compat_status != GTC_OK || !g_compat_ws) return g_compat_status;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return GTC_ERR_CUDA;
    std::lock_guard<std::mutex> lock(g_compat_mu);
    // the cached workspace was replaced by a later, larger call: its status
    // word belonged to that call
    if (g_compat[dev].ptr != g_compat_ws) return g_compat_status;
    unsigned int bits = 0;
    // a copy on the legacy default stream, so it waits for the count
    if (cudaMemcpy(&bits, g_compat_ws, sizeof(bits), cudaMemcpyDeviceToHost) != cudaSuccess)
        return GTC_ERR_CUDA;
    return status_from_bits(bits);
}

gtc_status gtc_count_status(const void *d_workspace, size_t ws_bytes, gtc_stream_t stream,
                            uint32_t *h_bits)
{
    if (!d_workspace || ws_bytes < sizeof(unsigned int)) return GTC_ERR_INVALID_ARGUMENT;
    unsigned int bits = 0;
    cudaStream_t s = as_stream(stream);
    if (cudaMemcpyAsync(&bits, d_workspace, sizeof(bits), cudaMemcpyDeviceToHost, s) != cudaSuccess)
        return GTC_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return GTC_ERR_CUDA;
    if (h_bits) *h_bits = bits;
    return status_from_bits(bits);
}

gtc_status gtc_compat_release(void)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return GTC_ERR_CUDA;
    std::lock_guard<std::mutex> lock(g_compat_mu);
    CompatCache &c = g_compat[dev];
    if (c.ptr) cudaFree(c.ptr);
    c.ptr = nullptr;
    c.bytes = 0;
    return GTC_OK;
}

void gtc_kernelCall_i64(unsigned int numberBlocks, unsigned int numberThreads, int64_t nv,
                        const int64_t *d_off, const int64_t *d_ind, int64_t *out,
                        int64_t threads_per_block, int64_t number_blocks, int64_t shifter)
{
    (void)numberBlocks; (void)threads_per_block; (void)number_blocks; (void)shifter;
    g_compat_status = GTC_OK;
    g_compat_ws = nullptr;
    if (!compat_block_size_ok(numberThreads)) { g_compat_status = GTC_ERR_INVALID_ARGUMENT; return; }
    if (nv <= 0 || !d_off || !out) { g_compat_status = GTC_ERR_INVALID_ARGUMENT; return; }
    int64_t nnz = 0;
    // the pipeline needs nnz = off[nv]: one 8-byte read on the legacy stream
    if (cudaMemcpy(&nnz, d_off + nv, sizeof(int64_t), cudaMemcpyDeviceToHost) != cudaSuccess) {
        g_compat_status = GTC_ERR_CUDA;
        return;
    }
    if (nnz < 0 || nv > 0x7fffffffll) { g_compat_status = GTC_ERR_INVALID_ARGUMENT; return; }
    size_t need = make_plan(nv, nnz, 64, true).bytes;
    size_t ind_bytes = (((size_t)nnz * sizeof(int)) + 255) & ~(size_t)255;
    char *ws = static_cast<char *>(compat_workspace(need + ind_bytes));
    if (!ws) { g_compat_status = GTC_ERR_OUT_OF_MEMORY; return; }
    int *ind32 = reinterpret_cast<int *>(ws + need);
    if (nnz > 0)
        narrow_kernel<<<(unsigned)div_up<long long>(nnz, 256), 256>>>(
            reinterpret_cast<const long long *>(d_ind), ind32, nnz, nv);
    const RowConfig cfg = pick_row_config(nv, nnz);
    g_compat_status = run_count<long long>(reinterpret_cast<const long long *>(d_off), ind32, nv,
                                           nnz, true, reinterpret_cast<long long *>(out), nullptr,
                                           nullptr, nullptr, ws, need, 0, cfg, nullptr);
    if (g_compat_status == GTC_OK) g_compat_ws = ws;
}

void gtc_kernelCall_i32(unsigned int numberBlocks, unsigned int numberThreads, int32_t nv,
                        const int32_t *d_off, const int32_t *d_ind, int32_t *out,
                        int32_t threads_per_block, int32_t number_blocks, int32_t shifter)
{
    (void)numberBlocks; (void)threads_per_block; (void)number_blocks; (void)shifter;
    g_compat_status = GTC_OK;
    g_compat_ws = nullptr;
    if (!compat_block_size_ok(numberThreads)) { g_compat_status = GTC_ERR_INVALID_ARGUMENT; return; }
    if (nv <= 0 || !d_off || !out) { g_compat_status = GTC_ERR_INVALID_ARGUMENT; return; }
    int32_t nnz = 0;
    if (cudaMemcpy(&nnz, d_off + nv, sizeof(int32_t), cudaMemcpyDeviceToHost) != cudaSuccess) {
        g_compat_status = GTC_ERR_CUDA;
        return;
    }
    if (nnz < 0) { g_compat_status = GTC_ERR_INVALID_ARGUMENT; return; }
    size_t need = make_plan(nv, nnz, 32, true).bytes;
    size_t r_bytes = (((size_t)nv * sizeof(long long)) + 255) & ~(size_t)255;
    char *ws = static_cast<char *>(compat_workspace(need + r_bytes));
    if (!ws) { g_compat_status = GTC_ERR_OUT_OF_MEMORY; return; }
    long long *r64 = reinterpret_cast<long long *>(ws + need);
    const RowConfig cfg = pick_row_config(nv, nnz);
    g_compat_status = run_count<int>(d_off, d_ind, nv, nnz, true, r64, nullptr, nullptr, nullptr,
                                     ws, need, 0, cfg, nullptr);
    if (g_compat_status == GTC_OK) {
        narrow_out_kernel<<<(unsigned)div_up<long long>(nv, 256), 256>>>(r64, out, nv);
        g_compat_ws = ws;
    }
}

void gtc_kernelCall_vertex_i64(unsigned int numberBlocks, unsigned int numberThreads, int64_t nv,
                               const int64_t *vertex, const int64_t *d_off, const int64_t *d_ind,
                               int64_t *out, int64_t threads_per_block, int64_t number_blocks,
                               int64_t shifter)
{
    (void)numberBlocks; (void)threads_per_block; (void)number_blocks; (void)shifter;
    g_compat_status = GTC_OK;
    g_compat_ws = nullptr;
    if (!compat_block_size_ok(numberThreads)) { g_compat_status = GTC_ERR_INVALID_ARGUMENT; return; }
    if (nv < 0 || (nv > 0 && (!vertex || !d_off || !d_ind || !out))) {
        g_compat_status = GTC_ERR_INVALID_ARGUMENT;
        return;
    }
    g_compat_status = launch_subset(reinterpret_cast<const long long *>(d_off),
                                    reinterpret_cast<const long long *>(d_ind),
                                    reinterpret_cast<const long long *>(vertex), nv,
                                    reinterpret_cast<long long *>(out), 0);
}

void gtc_kernelCall_vertex_i32(unsigned int numberBlocks, unsigned int numberThreads, int32_t nv,
                               const int32_t *vertex, const int32_t *d_off, const int32_t *d_ind,
                               int32_t *out, int32_t threads_per_block, int32_t number_blocks,
                               int32_t shifter)
{
    (void)numberBlocks; (void)threads_per_block; (void)number_blocks; (void)shifter;
    g_compat_status = GTC_OK;
    g_compat_ws = nullptr;
    if (!compat_block_size_ok(numberThreads)) { g_compat_status = GTC_ERR_INVALID_ARGUMENT; return; }
    if (nv < 0 || (nv > 0 && (!vertex || !d_off || !d_ind || !out))) {
        g_compat_status = GTC_ERR_INVALID_ARGUMENT;
        return;
    }
    g_compat_status = launch_subset(d_off, d_ind, vertex, (long long)nv, out, 0);
}

}  // extern "C"
