// gtc_internal.cuh -- shared device/host helpers of the B200 triangle counter.
//
// Algorithm (same output as the reference's per-vertex kernel,
// src/clusteringCount.cu:314-359, computed differently):
//   1. order the vertices by degree and orient every undirected edge from its
//      lower to its higher end; N+(v), v's forward list, is written to the
//      start of v's own CSR segment in one pass.  The vertices of the highest
//      degrees -- the core, a set closed upwards in the order -- are numbered
//      by a counting sort of their degrees (position 0 = highest) and named by
//      position; every other vertex keeps its id;
//   2. the core's forward lists become the rows of a triangular bit matrix U:
//      bit s of row q is set iff q -> s;
//   3. every triangle p < q < s is found at its lowest vertex p, at the edge
//      p -> q.  If q is a core vertex then so is s, and the pair (q, s) of
//      N+(p) is tested in U, one bit per pair.  Otherwise q's forward list is
//      looked up in a shared-memory table of N+(p);
//   4. the triangle is credited to p, q and s: p by a sum, q by a population
//      count, s by a per-member counter, each flushed once per (p, member).
// All counting is integer and exact; the result does not depend on the order
// in which blocks run nor on the order of equal degrees.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/gtc_b200.h"

namespace gtc {

// ------------------------------------------------------------------ tuning
constexpr int kThreads = 256;               // every pipeline kernel
// Vertices from which lists and core pairs get a kernel each: R-MAT 17 takes
// 193 us in one kernel and 211 in two, R-MAT 20 of mean degree 16 (global count)
// 656 and 618; R-MAT 18 and 19 of 16, in between, 228 and 253, 396 and 407.
constexpr long long kSmallGraph = 1ll << 18;
constexpr int kShortRow = 64;               // longest row placed with its neighbours
// Longest forward list of a short row; of a uniform graph.  16 instead of 32:
// R-MAT 20 1507 us instead of 1519, but the 512-graph batch 11.4 ms instead of
// 10.6.  32 instead of 64: ER 900K of mean degree 30 400 us instead of 346.
constexpr int kShortList = 32;
constexpr int kShortListIds = 64;
constexpr int kRowChunk = 256;              // entries of a longer row per placement item
constexpr int kBuckets = 1024;              // degree buckets (counting sort of the core)
constexpr int kCoreMax = 32768;             // most core vertices of a graph
constexpr int kCoreMinDegree = kShortRow + 1;   // core rows are never short rows
constexpr int kCoreDegreeRatio = 2, kCoreDegreeOver = 16;   // ... of this multiple of the mean, plus
constexpr int kMemberChunk = 1024;          // members of a wide row held at a time
constexpr int kTableLog2 = 12;              // wide rows: shared hash slots
constexpr int kKeyTop = 0x7fffffff;         // key of core position 0
constexpr int kNoMember = INT32_MIN;        // never a list element

// Error bits written to the workspace status word (the first 4 bytes of
// every counting workspace) by device code; gtc_count_status reads them.
enum : unsigned int {
    kErrIndexRange = 1u,   // a neighbour id outside [0, n) was met (and skipped)
};

// Per-vertex record: forward-list start, forward degree and the number of
// core members, in one 16-byte load.  kWideRow in dk marks rows that a warp or a
// block takes alone (core rows, rows longer than kShortRow, forward lists longer
// than kShortList); those are the wide list.
constexpr int kWideRow = INT32_MIN;
struct __align__(16) VInfo {
    long long fbeg;
    int fdeg;
    int dk;
};

// GraphRec::uniform of a graph whose rows have signatures (Sign).
constexpr int kSigned = 2, kSigWords = 8;
constexpr int kSignedGraph = 512;           // vertices of the smallest such graph,
constexpr int kSignedCall = 32768;          // ... of the smallest call (all its graphs)

// Per-graph record (one for a single graph, one per graph of a batch).
struct GraphRec {
    long long v0 = 0;          // first vertex
    long long ubase = 0;       // first word of the graph's bit matrix, or of its signatures in find
    int nv = 0;                // vertices
    int core = 0;              // core vertices K
    int min_bucket = kBuckets; // lowest degree bucket of the core
    int dmin = 0;              // lowest degree that may be core
    int long_min = 0;          // rows longer than this are placed by blocks
    int kcap = 0;              // most core vertices (bit-matrix space)
    int uniform = 0;           // no vertex of core degree: rows ordered by id; kSigned too
};

// Counters block in the workspace (device, zeroed at the start of a count).
struct Counters {
    unsigned long long tri_total;     // triangles found (T)
    unsigned long long wide_rows;     // entries of the wide list
    unsigned long long place_items;   // placement items posted for long rows
    unsigned long long place_next;    // dynamic queues:
    unsigned long long core_long_next, core_wide_next, core_short_next;
    unsigned long long table_long_next, table_wide_next, list_short_next;
    unsigned long long bitmap_next;
    unsigned long long u_words;       // bit-matrix words handed out (batch)
    unsigned int blocks_done;         // degree pass: blocks finished
};

__host__ __device__ constexpr int ilog2(int v) { return v <= 1 ? 0 : 1 + ilog2(v >> 1); }

// Monotone map of a degree onto kBuckets buckets: exact below half of them,
// then kBuckets / 32 buckets per octave -- a float with 5 mantissa bits -- for
// the next 16 octaves, the rest in the last bucket.
__host__ __device__ __forceinline__ int degree_bucket(int d)
{
    constexpr int kExact = kBuckets / 2, kPer = kBuckets / 32;
    constexpr int kLe = ilog2(kExact), kMb = ilog2(kPer);
    if (d < kExact) return d < 0 ? 0 : d;
    int l = kLe;
    while ((d >> (l + 1)) != 0) ++l;
    const int b = kExact + (l - kLe) * kPer + ((d >> (l - kMb)) & (kPer - 1));
    return b < kBuckets ? b : kBuckets - 1;
}

// First word of core row `pos` in the triangular bit matrix; u_row(K) is the
// size of a K-row matrix.  Row pos holds bits [0, pos) in whole 32-byte
// sectors: 8 * (pos / 256 + 1) words.
__host__ __device__ __forceinline__ int u_row(int pos)
{
    const int a = pos >> 8;
    return 8 * (a + 1) * (128 * a + (pos & 255));
}

__device__ __forceinline__ unsigned int hash_slot(int key, int log2_slots)
{
    return ((unsigned int)key * 0x9E3779B1u) >> (32 - log2_slots);
}

// What a member sets in its row's signature: three bits of one word, one in
// each third of its low 30.  A row of 15 members lets one in a hundred ids pass
// that are none of them; with one bit anywhere in the 256 it was one in 17.
struct Sign {
    int word;
    unsigned int bits;
};

__device__ __forceinline__ Sign sign_of(int y)
{
    const unsigned int h = (unsigned int)y * 0x9E3779B1u;
    const unsigned int a = (h >> 21 & 0xff) * 10 >> 8, b = (h >> 13 & 0xff) * 10 >> 8,
                       c = (h >> 5 & 0xff) * 10 >> 8;
    return {(int)(h >> 29), (1u << a) | (0x400u << b) | (0x100000u << c)};
}

__host__ __device__ __forceinline__ int ceil_log2(long long v)
{
    int l = 0;
    while ((1ll << l) < v) ++l;
    return l;
}

template <typename T>
__host__ __device__ __forceinline__ T div_up(T a, T b)
{
    return (a + b - 1) / b;
}

}  // namespace gtc
