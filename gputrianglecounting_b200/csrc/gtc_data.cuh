// gtc_data.cuh -- what the kernels of one count share: the arrays they read
// and write, and warp-level helpers.
#pragma once

#include "gtc_internal.cuh"

namespace gtc {

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
    int *wide;                      // rows that a warp or a block takes alone
    int2 *litem;                    // placement items of long rows: {row, chunk}
    unsigned int *u;                // bit matrices
    long long ucap;                 // words of it
    unsigned long long *tacc;       // t(v) without the core's credits (null: global count only)
    unsigned long long *tcore;      // credits of core vertices: [first vertex + position]
    unsigned long long *gsum;       // batch: sum of t per graph
    Counters *ctr;
    unsigned int *status;
    int word;                       // sizeof(unsigned int)
    const int *gate;                // nullable: while it is 0 the kernels end at once
    bool bitmaps, sparse;           // bitmap_kernel runs too; sparse_core_kernel for core_kernel
};
template <typename OffT>
struct View : Data {
    const OffT *off;
};

__device__ __forceinline__ bool gated(const Data &w) { return w.gate && !*w.gate; }

__device__ __forceinline__ int warp_incl_scan(int v)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += o;
    }
    return v;
}

// The lane i whose [incl_i - count_i, incl_i) holds f (incl: this lane's
// inclusive prefix of a per-lane count).
__device__ __forceinline__ int warp_corank(int incl, int f)
{
    int i = 0;
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
        const int v = __shfl_sync(0xffffffffu, incl, i + step - 1);
        if (v <= f) i += step;
    }
    return i;
}

}  // namespace gtc
