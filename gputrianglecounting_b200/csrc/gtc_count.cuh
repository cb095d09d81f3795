// gtc_count.cuh -- kernels that find the triangles: pairs of core members in
// the bit matrix, forward lists of the other members in hash tables; and the
// epilogue.
#pragma once

#include <cuda_pipeline.h>

#include "gtc_build.cuh"

namespace gtc {

__device__ __forceinline__ void add64(unsigned long long *p, unsigned int x)
{
    atomicAdd(p, (unsigned long long)x);
}

__device__ __forceinline__ unsigned int warp_sum(unsigned int x)
{
    return __reduce_add_sync(0xffffffffu, x);
}

// A lane's constants of the 32 x 32 bit transpose.  They are kept (the
// compiler is not to derive them anew for every transpose).
struct Transposer {
    unsigned int sel16, sel8, keep4, keep2, keep1;
    int rot4, rot2, rot1;

    static __device__ __forceinline__ unsigned int held(unsigned int x)
    {
        unsigned int y;
        asm volatile("mov.b32 %0, %1;" : "=r"(y) : "r"(x));
        return y;
    }
    __device__ __forceinline__ explicit Transposer(int lane)
    {
        sel16 = held(lane & 16 ? 0x3276 : 0x5410);
        sel8 = held(lane & 8 ? 0x3715 : 0x6240);
        keep4 = held(lane & 4 ? 0xf0f0f0f0u : 0x0f0f0f0fu);
        keep2 = held(lane & 2 ? 0xccccccccu : 0x33333333u);
        keep1 = held(lane & 1 ? 0xaaaaaaaau : 0x55555555u);
        rot4 = (int)held(lane & 4 ? 28 : 4);
        rot2 = (int)held(lane & 2 ? 30 : 2);
        rot1 = (int)held(lane & 1 ? 31 : 1);
    }
    // Bit c of lane r's result is bit r of lane c's x.  At distance k the lanes
    // swap the halves of every 2k-bit field; a rotation by k (back for the upper
    // lanes) aligns the partner's bits.
    __device__ __forceinline__ unsigned int operator()(unsigned int x) const
    {
        x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 16), sel16);
        x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 8), sel8);
        unsigned int y = __shfl_xor_sync(0xffffffffu, x, 4);
        x = (x & keep4) | (__funnelshift_l(y, y, rot4) & ~keep4);
        y = __shfl_xor_sync(0xffffffffu, x, 2);
        x = (x & keep2) | (__funnelshift_l(y, y, rot2) & ~keep2);
        y = __shfl_xor_sync(0xffffffffu, x, 1);
        return (x & keep1) | (__funnelshift_l(y, y, rot1) & ~keep1);
    }
};

// Credit of a list element: vertices in tacc, core positions in tcore.
__device__ __forceinline__ void credit(const Data &w, long long v0, int shift, int m,
                                       unsigned int c)
{
    add64(m >= 0 ? &w.tacc[m + shift] : &w.tcore[v0 + ~m], c);
}

// ============================================== pairs of core members (bits)

// base[i], the address in one multiply-add: the integer pipe that adds and
// shifts is the busy one here, and a multiplier `word` (4) that the compiler
// cannot see keeps the address off it.
__device__ __forceinline__ unsigned int load_word(const unsigned int *base, int i, int word)
{
    unsigned long long p;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(p) : "r"(i), "r"(word), "l"(base));
    return __ldg(reinterpret_cast<const unsigned int *>(p));
}

// A core member s as a lane sees it: its word in row 0, and the factor that
// moves its bit to the top.
struct CoreBit {
    const unsigned int *up;
    unsigned int mul;
};

__device__ __forceinline__ CoreBit core_bit(const unsigned int *U, int pos)
{
    return {U + (pos >> 5), 0x80000000u >> (pos & 31)};
}

// Bit k of the result: whether s is in core row k of qb[0 .. nq) (word
// offsets; entries up to the next multiple of 16 must be readable).  Per row
// an address, a load, a multiplication that brings the bit to the top, a shift
// that takes it in and a quarter of a shared load; 16 loads in flight.
__device__ __forceinline__ unsigned int row_bits(const CoreBit &s, const int *qb, int nq, int word)
{
    unsigned int hb = 0;
    int i = 0;
    for (; i < nq; i += 16) {
        unsigned int x[16];
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
            const int4 a = *reinterpret_cast<const int4 *>(qb + i + j);
            x[j] = load_word(s.up, a.x, word);
            x[j + 1] = load_word(s.up, a.y, word);
            x[j + 2] = load_word(s.up, a.z, word);
            x[j + 3] = load_word(s.up, a.w, word);
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            unsigned int t;
            asm("mul.lo.u32 %0, %1, %2;" : "=r"(t) : "r"(x[j]), "r"(s.mul));
            hb = __funnelshift_l(t, hb, 1);
        }
    }
    hb = __brev(hb) >> (32 - i);                  // i >= 16; row k at bit k
    return nq < 32 ? hb & ((1u << nq) - 1u) : hb;
}

// Ascending sort of 32 E integers by a warp in registers (bitonic network):
// lane l ends with elements l E .. l E + E - 1.
template <int E>
__device__ __forceinline__ void warp_sort(int (&v)[E], int lane)
{
#pragma unroll
    for (int k = 2; k <= 32 * E; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= E) {
                const bool lower = (lane & (j / E)) == 0;
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const bool asc = k >= E ? (lane & (k / E)) == 0 : (e & k) == 0;
                    const int y = __shfl_xor_sync(0xffffffffu, v[e], j / E);
                    v[e] = lower == asc ? min(v[e], y) : max(v[e], y);
                }
            } else {
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    if ((e & j) == 0) {
                        const bool asc = k >= E ? (lane & (k / E)) == 0 : (e & k) == 0;
                        const int a = v[e], b = v[e + j];
                        v[e] = asc ? min(a, b) : max(a, b);
                        v[e + j] = asc ? max(a, b) : min(a, b);
                    }
                }
            }
        }
    }
}

// Whose first share this block takes of the second and third kind of work of
// a kernel.  With less than two rows per warp most blocks have no other share,
// and those that took wide rows should not have the first tiles too (R-MAT 10,
// counting kernel: 13.9 us all from block 0 on, 12.4 shifted); with more the
// blocks come free at different times (R-MAT 17: 127 us, 134 shifted).
__device__ __forceinline__ long long first_block(long long n, unsigned int shift)
{
    const bool few = n < 2ll * gridDim.x * (kThreads / 32);
    return few ? (blockIdx.x + shift) % gridDim.x : blockIdx.x;
}

// Longest list of a wide row that a warp takes: bit matrix, tables (tables of
// 256 members for a warp, half full: R-MAT 22's wide rows 5300 us against 4726).
constexpr int kWarpList = 256, kWarpTable = 128;
constexpr int kClaim = 128;                       // most wide rows a block looks through at a time
constexpr int kWarpClaim = 8;                     // ... a warp

// A block's share of the wide list's long rows.
struct WideClaim {
    int row[kClaim];
    int count;
    long long item;
};

// The rows of the wide list of more than `most` members that `want` (of the
// row's record), each by a whole block (by_block).  First shares are fixed, the
// next ones come from a queue.  A share's rows are spread over the list, whose
// neighbours tend to be alike (generators give hubs the lowest ids).
template <class Want, class ByBlock>
__device__ __forceinline__ void wide_block_rows(const Data &w, WideClaim &cl, long long block,
                                                unsigned long long *long_next, int most,
                                                const Want &want, const ByBlock &by_block)
{
    const long long rows = (long long)w.ctr->wide_rows;
    // shares small enough that the last ones leave no long tail
    const int per_block = (int)min((long long)kClaim, max(8ll, rows / (4ll * gridDim.x)));
    const long long claims = div_up<long long>(rows, per_block);
    long long item = block;
    while (item < claims) {
        __syncthreads();
        if (threadIdx.x == 0) cl.count = 0;
        __syncthreads();
        if (threadIdx.x < per_block && item + claims * threadIdx.x < rows) {
            const int v = w.wide[item + claims * threadIdx.x];
            const VInfo vi = w.vinfo[v];
            if (vi.fdeg > most && want(vi)) cl.row[atomicAdd(&cl.count, 1)] = v;
        }
        __syncthreads();
        for (int k = 0; k < cl.count; ++k) {
            const int v = cl.row[k];
            by_block(v, w.vinfo[v]);
        }
        if (gridDim.x >= claims) break;
        __syncthreads();
        if (threadIdx.x == 0) cl.item = gridDim.x + (long long)atomicAdd(long_next, 1ull);
        __syncthreads();
        item = cl.item;
    }
}

// The same, and those of at most `most` members by a warp each (by_warp).
template <class Want, class ByBlock, class ByWarp>
__device__ __forceinline__ void wide_rows(const Data &w, WideClaim &cl, long long block,
                                          unsigned long long *long_next,
                                          unsigned long long *next, int most, const Want &want,
                                          const ByBlock &by_block, const ByWarp &by_warp)
{
    wide_block_rows(w, cl, block, long_next, most, want, by_block);
    __syncthreads();
    const long long rows = (long long)w.ctr->wide_rows;
    const int lane = threadIdx.x & 31;
    const long long warps = (long long)gridDim.x * (kThreads / 32);
    const int per_warp = (int)min((long long)kWarpClaim, max(1ll, rows / (16 * warps)));
    const long long claims = div_up<long long>(rows, per_warp);
    long long item = block * (kThreads / 32) + (threadIdx.x >> 5);
    while (item < claims) {
        const long long at = item + claims * lane;
        int v = 0;
        VInfo vi{0, 0, 0};
        bool in = lane < per_warp && at < rows;
        if (in) {
            v = w.wide[at];
            vi = w.vinfo[v];
            in = vi.fdeg <= most && want(vi);
        }
        unsigned int todo = __ballot_sync(0xffffffffu, in);
        while (todo) {
            const int k = __ffs(todo) - 1;
            todo &= todo - 1;
            by_warp(__shfl_sync(0xffffffffu, v, k),
                    VInfo{__shfl_sync(0xffffffffu, vi.fbeg, k),
                          __shfl_sync(0xffffffffu, vi.fdeg, k),
                          __shfl_sync(0xffffffffu, vi.dk, k)});
        }
        if (warps >= claims) break;
        if (lane == 0) item = warps + (long long)atomicAdd(next, 1ull);
        item = __shfl_sync(0xffffffffu, item, 0);
    }
}

struct CoreWarpSmem {
    int qb[kWarpList];                            // word offset of each member's core row
    unsigned int cnt[kWarpList];
    unsigned short pos[kWarpList];
};

struct CoreBlockSmem {
    unsigned int bits[kCoreMax / 32];             // the row's core members
    unsigned short below[kCoreMax / 32];          // members in earlier words
    int spos[kMemberChunk], qpos[kMemberChunk];   // positions of the s and q members
    int qb[kMemberChunk];                         // word offset of each q member's row
    unsigned int scnt[kMemberChunk], qcnt[kMemberChunk];
    unsigned int wsum[kThreads / 32];
    unsigned int total;
};

struct CoreSmem {
    union {
        CoreWarpSmem warp[kThreads / 32];
        CoreBlockSmem block;
    };
    WideClaim claim;
};

// Where a row's core lives.
struct CoreView {
    const unsigned int *U;
    unsigned long long *tcore;
    unsigned long long *own;      // the row's own credits
};

template <bool PV, bool BATCH>
__device__ __forceinline__ CoreView core_view(const Data &w, int v)
{
    const GraphRec *rec = &w.recs[BATCH ? w.gid[v] : 0];
    CoreView c{w.u, w.tcore, nullptr};
    if (BATCH) {
        c.U += rec->ubase;
        c.tcore += rec->v0;
    }
    if (PV) {
        const int kv = w.key[v];
        c.own = kv > kKeyTop - rec->core ? &c.tcore[kKeyTop - kv] : &w.tacc[v];
    }
    return c;
}

// Pairs (q, s) of core members of one row, q -> s a bit of U: with the members
// in ascending position (descending order) s has the lower index, so the pairs
// are a lower triangle of index pairs, in tiles of 32 q by 32 s.  A lane holds
// a member s and loads its word of 32 rows q.  A tile's hits are a 32 x 32 bit
// matrix: rows count s, columns (transposed) count q.  Waits for the gathered
// words bound it, then L1 wavefronts (71%), at 32 warps per SM and 64 registers
// (R-MAT 20, 1.19e9 pairs, wide rows: 781 us; five blocks of 48 registers 1053
// when this took 946; looking ids up in shared tables of the longer lists,
// which this replaced, 2375).

// A row of at most kWarpList members (32 E) by a warp, sorted in registers.
template <int E, bool PV>
__device__ __forceinline__ void core_warp_row(const Data &w, const VInfo &vi, const CoreView &cv,
                                              const Transposer &tr, CoreWarpSmem &sm,
                                              unsigned long long &tri)
{
    const int lane = threadIdx.x & 31;
    int p[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int k = e * 32 + lane;
        const int m = k < vi.fdeg ? w.find[vi.fbeg + k] : 0;
        p[e] = m < 0 ? ~m : INT32_MAX;
    }
    warp_sort<E>(p, lane);
    const int n = vi.dk & INT32_MAX;
    __syncwarp();
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int k = lane * E + e;
        sm.pos[k] = (unsigned short)p[e];
        sm.qb[k] = k < n ? u_row(p[e]) : 0;
        if (PV) sm.cnt[k] = 0;
    }
    __syncwarp();
    unsigned int tot = 0;
    const int groups = (n + 31) >> 5;
    for (int ts = 0; ts < groups; ++ts) {
        const int si = ts * 32 + lane;
        const CoreBit s = core_bit(cv.U, si < n ? sm.pos[si] : 0);
        // s is above q only at lower indices
        unsigned int keep = si < n && lane < 31 ? 0xffffffffu << (lane + 1) : 0u, v = 0;
        for (int tq = ts; tq < groups; ++tq) {
            const unsigned int hb = keep & row_bits(s, sm.qb + tq * 32, min(32, n - tq * 32),
                                                    w.word);
            keep = 0xffffffffu;
            v += __popc(hb);
            // an index modulo 32 belongs to one lane
            if (PV) sm.cnt[tq * 32 + lane] += __popc(tr(hb));
        }
        tot += v;
        if (PV) sm.cnt[si] += v;
    }
    tot = warp_sum(tot);
    if (tot) {
        if (PV) {
            for (int k = lane; k < n; k += 32)
                if (sm.cnt[k]) add64(&cv.tcore[sm.pos[k]], sm.cnt[k]);
            if (lane == 0) add64(cv.own, tot);
        }
        tri += lane == 0 ? tot : 0u;
    }
}

// A longer row by the block: a bitmap of the members over the core positions
// and the members below each of its words give every member its index; rows
// of more than kMemberChunk members go chunk by chunk.
template <bool PV>
__device__ void core_block_row(const Data &w, const VInfo &vi, int core, const CoreView &cv,
                               const Transposer &tr, CoreBlockSmem &sm, unsigned long long &tri)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int words = (core + 31) >> 5;
    constexpr int kPer = kCoreMax / 32 / kThreads;
    __syncthreads();
    for (int k = threadIdx.x; k < kThreads * kPer; k += kThreads) sm.bits[k] = 0;
    if (threadIdx.x == 0) sm.total = 0;
    __syncthreads();
    for (int k = threadIdx.x; k < vi.fdeg; k += kThreads) {
        const int m = w.find[vi.fbeg + k];
        if (m < 0) atomicOr(&sm.bits[~m >> 5], 1u << (~m & 31));
    }
    __syncthreads();
    const int w0 = threadIdx.x * kPer;
    int cnt[kPer], sum = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        cnt[j] = __popc(sm.bits[w0 + j]);
        sum += cnt[j];
    }
    int incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
    }
    if (lane == 31) sm.wsum[warp] = (unsigned int)incl;
    __syncthreads();
    int first = incl - sum, total = 0;
    for (int i = 0; i < kThreads / 32; ++i) {
        if (i < warp) first += (int)sm.wsum[i];
        total += (int)sm.wsum[i];
    }
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        if (w0 + j < words) sm.below[w0 + j] = (unsigned short)first;
        first += cnt[j];
    }
    __syncthreads();
    auto fill = [&](int base, int *pos, int *qb) {
        for (int k = threadIdx.x; k < vi.fdeg; k += kThreads) {
            const int m = w.find[vi.fbeg + k];
            if (m >= 0) continue;
            const int x = ~m;
            const int at = sm.below[x >> 5] +
                           __popc(sm.bits[x >> 5] & ((1u << (x & 31)) - 1u)) - base;
            if (at >= 0 && at < kMemberChunk) {
                pos[at] = x;
                if (qb) qb[at] = u_row(x);
            }
        }
        if (qb)
            for (int k = total - base + (int)threadIdx.x;
                 k < kMemberChunk && k < total - base + 16; k += kThreads)
                qb[k] = 0;
    };
    unsigned int mine = 0;
    const bool one = total <= kMemberChunk;
    for (int sb = 0; sb < total; sb += kMemberChunk) {
        const int ns = min(total - sb, kMemberChunk), sg = (ns + 31) >> 5;
        fill(sb, sm.spos, one ? sm.qb : nullptr);
        if (PV)
            for (int k = threadIdx.x; k < ns; k += kThreads) sm.scnt[k] = 0;
        for (int qs = sb; qs < total; qs += kMemberChunk) {
            const int nq = min(total - qs, kMemberChunk), qg = (nq + 31) >> 5;
            if (!one) fill(qs, sm.qpos, sm.qb);
            if (PV)
                for (int k = threadIdx.x; k < nq; k += kThreads) sm.qcnt[k] = 0;
            __syncthreads();
            const bool diag = qs == sb;
            // tiles, the q groups of an s group in turn, parted evenly among
            // the warps
            const int tiles = diag ? qg * (qg + 1) / 2 : qg * sg;
            const int t1 = tiles * (warp + 1) / (kThreads / 32);
            int t = tiles * warp / (kThreads / 32), ts, tq;
            if (diag) {                           // from the last tile, a triangle row by row
                const int r = tiles - 1 - t;
                int a = (int)((sqrtf(8.0f * (float)r + 1.0f) - 1.0f) * 0.5f);
                while (a * (a + 1) / 2 > r) --a;
                while ((a + 1) * (a + 2) / 2 <= r) ++a;
                ts = qg - 1 - a;
                tq = qg - 1 - (r - a * (a + 1) / 2);
            } else {
                ts = t / qg;
                tq = t - ts * qg;
            }
            while (t < t1) {
                const int si = ts * 32 + lane;
                const CoreBit s = core_bit(cv.U, si < ns ? sm.spos[si] : 0);
                unsigned int v = 0;
                for (; tq < qg && t < t1; ++tq, ++t) {
                    unsigned int hb = row_bits(s, sm.qb + tq * 32, min(32, nq - tq * 32), w.word);
                    if (diag && tq == ts) hb &= lane < 31 ? 0xffffffffu << (lane + 1) : 0u;
                    if (si >= ns) hb = 0;
                    v += __popc(hb);
                    if (PV) {
                        const unsigned int c = __popc(tr(hb));
                        if (c) atomicAdd(&sm.qcnt[tq * 32 + lane], c);
                    }
                }
                if (PV) {
                    if (v) atomicAdd(&sm.scnt[si], v);
                } else {
                    mine += v;
                }
                ++ts;
                tq = diag ? ts : 0;
            }
            __syncthreads();
            if (PV) {
                const int *pos = one ? sm.spos : sm.qpos;
                for (int k = threadIdx.x; k < nq; k += kThreads) {
                    const unsigned int c = sm.qcnt[k];
                    mine += c;
                    const unsigned int both = one ? c + sm.scnt[k] : c;
                    if (both) add64(&cv.tcore[pos[k]], both);
                }
                __syncthreads();
            }
        }
        if (PV && !one) {
            for (int k = threadIdx.x; k < ns; k += kThreads)
                if (sm.scnt[k]) add64(&cv.tcore[sm.spos[k]], sm.scnt[k]);
            __syncthreads();
        }
    }
    // at most kCoreMax members: their pairs, 2^29, fit 32 bits
    const unsigned int ws = warp_sum(mine);
    if (lane == 0 && ws) atomicAdd(&sm.total, ws);
    __syncthreads();
    if (threadIdx.x == 0 && sm.total) {
        if (PV) add64(cv.own, sm.total);
        tri += sm.total;
    }
}

template <bool PV, bool BATCH>
__device__ __forceinline__ void core_wide_rows(const Data &w, CoreSmem &sm,
                                               unsigned long long &tri)
{
    const Transposer tr(threadIdx.x & 31);
    wide_rows(
        w, sm.claim, blockIdx.x, &w.ctr->core_long_next, &w.ctr->core_wide_next, kWarpList,
        [](const VInfo &vi) { return (vi.dk & INT32_MAX) >= 2; },
        [&](int v, const VInfo &vi) {
            core_block_row<PV>(w, vi, w.recs[BATCH ? w.gid[v] : 0].core,
                               core_view<PV, BATCH>(w, v), tr, sm.block, tri);
        },
        [&](int v, const VInfo &vi) {
            const CoreView cv = core_view<PV, BATCH>(w, v);
            CoreWarpSmem &ws = sm.warp[threadIdx.x >> 5];
            if (vi.fdeg <= 32) core_warp_row<1, PV>(w, vi, cv, tr, ws, tri);
            else if (vi.fdeg <= 64) core_warp_row<2, PV>(w, vi, cv, tr, ws, tri);
            else if (vi.fdeg <= 128) core_warp_row<4, PV>(w, vi, cv, tr, ws, tri);
            else core_warp_row<8, PV>(w, vi, cv, tr, ws, tri);
        });
}

// Short rows of at most W members, 32 / W at a time, W lanes each: a lane per
// member, every core member q of a row in turn tested against the core members
// above it, four q in flight.
template <int W, bool PV, bool BATCH>
__device__ __forceinline__ void core_rows(const Data &w, long long u0, const VInfo &vi, int g,
                                          unsigned int rows, unsigned long long &tri)
{
    constexpr int kGroups = 32 / W;
    const int lane = threadIdx.x & 31, grp = lane / W, gl = lane % W, g0 = grp * W;
    const unsigned int gmask = (W == 32 ? 0xffffffffu : (1u << W) - 1u) << g0;
    while (rows) {
        int r = -1;
#pragma unroll
        for (int k = 0; k < kGroups; ++k) {
            if (k == grp && rows) r = __ffs(rows) - 1;
            rows &= rows - 1;
        }
        const long long fb = __shfl_sync(0xffffffffu, vi.fbeg, r & 31);
        const int fd = __shfl_sync(0xffffffffu, vi.fdeg, r & 31);
        const int m = r >= 0 && gl < fd ? w.find[fb + gl] : 0;
        const bool core = m < 0;
        const int pos = ~m;
        const int rb = core ? u_row(pos) : INT32_MAX;   // ascending with the position
        const unsigned int *up = w.u + (core ? pos >> 5 : 0);
        long long v0 = 0;
        if (BATCH) {
            const GraphRec *rec = &w.recs[__shfl_sync(0xffffffffu, g, r & 31)];
            up += rec->ubase;
            v0 = rec->v0;
        }
        unsigned int qm = __ballot_sync(0xffffffffu, core) & gmask;
        unsigned int cq = 0, cs = 0;
        while (__any_sync(0xffffffffu, qm != 0)) {
            int q[4];
            unsigned int x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                q[j] = __ffs(qm) - 1;
                qm &= qm - 1;
                const int rq = __shfl_sync(0xffffffffu, rb, q[j] & 31);
                x[j] = q[j] >= 0 && rb < rq ? __ldg(up + rq) : 0u;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool hit = (x[j] >> (pos & 31)) & 1u;
                const unsigned int h = __ballot_sync(0xffffffffu, hit) & gmask;
                cs += hit;
                if (lane == q[j]) cq += __popc(h);
            }
        }
        unsigned int tot = cq;
#pragma unroll
        for (int d = W / 2; d > 0; d >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, d);
        if (PV) {
            if (core && cq + cs) add64(&w.tcore[v0 + pos], cq + cs);
            if (gl == 0 && tot) add64(&w.tacc[u0 + r], tot);
        }
        tri += gl == 0 ? tot : 0u;
    }
}

template <bool PV, bool BATCH>
__device__ __forceinline__ void core_short_rows(const Data &w, long long u0, int batch,
                                                unsigned long long &tri)
{
    const int lane = threadIdx.x & 31;
    VInfo vi{0, 0, 0};
    int g = 0;
    if (lane < batch && u0 + lane < w.n) {
        vi = w.vinfo[u0 + lane];
        if (BATCH) g = w.gid[u0 + lane];
    }
    const bool act = vi.dk >= 2;                  // not a wide row
    const unsigned int narrow = __ballot_sync(0xffffffffu, act && vi.fdeg <= 8);
    const unsigned int mid = __ballot_sync(0xffffffffu, act && vi.fdeg > 8 && vi.fdeg <= 16);
    const unsigned int full = __ballot_sync(0xffffffffu, act && vi.fdeg > 16);
    if (narrow) core_rows<8, PV, BATCH>(w, u0, vi, g, narrow, tri);
    if (mid) core_rows<16, PV, BATCH>(w, u0, vi, g, mid, tri);
    if (full) core_rows<32, PV, BATCH>(w, u0, vi, g, full, tri);
}

// ====================================================== other members (lists)

constexpr int kNoProbe = INT32_MIN + 1;           // never a list element nor kNoMember

// A tile: consecutive short rows with at most kTileEdges members in all, of
// which at most kTileIds are distinct.
constexpr int kTileEdges = 192, kTileIds = 96, kTileWords = kTileIds / 32;
constexpr int kTileSlots = 2048;
constexpr int kTileLong = 32;                     // longer lists are taken by the whole warp
constexpr int kNoId = 0xff, kClaimed = 0x80;      // a slot that is empty, that a lane claims

// Of SignedRows: rows' members, their signatures, pairs to search for.
constexpr int kPairs = 64;

struct SignedSmem {
    unsigned int sign[2][kSigWords * 35];         // 32 signatures and a gap between four groups
    int member[2][32];
    int q[kPairs], s[kPairs];
    unsigned char row[kPairs];
};

template <typename Pos>
struct TileData {
    unsigned int adj[kTileWords][kTileIds];       // adjacency among the tile's distinct members
    unsigned int rowbits[kTileWords][32];         // a row's members
    Pos start[kTileIds];                          // a streamed list's begin, less its elements before
    union {
        unsigned int begins[kTileIds];            // bit f: a list begins at element f of the stream
        unsigned int credit[kTileIds];
    };
    int member[kTileIds];                         // a number's member
    unsigned short edge[kTileEdges];              // the number of an edge's member, its row << 8
    unsigned char owner[kTileIds];                // number whose list is the k-th of the stream
    unsigned char from[32];                       // lane of the k-th row that takes part
};

template <typename Pos>
struct __align__(16) TileSmem {
    unsigned char slot[kTileSlots];               // number of the member that hashes here
    union {
        TileData<Pos> tile;
        SignedSmem sign;
    };
};
static_assert(kTileLong * kTileIds <= 32 * kTileIds, "begins holds a bit per streamed element");
static_assert(kTileIds <= kClaimed, "numbers and claims share a byte");

// Empties a warp's table; every tile leaves it empty again.
template <typename Pos>
__device__ __forceinline__ void tile_init(TileSmem<Pos> &sm)
{
    for (int k = threadIdx.x & 31; k < kTileSlots / 4; k += 32)
        reinterpret_cast<unsigned int *>(sm.slot)[k] = 0xffffffffu;
    __syncwarp();
}

// Short rows, a tile at a time by a warp.  The members of all rows of the
// tile are numbered through a shared hash table (rows near each other share
// members: on a geometric graph a tile's 160 edges have some 75), every
// distinct member's forward list is looked up once -- all lists as one stream,
// so that every lane has an element -- and what is found sets the bits of the
// symmetric adjacency among the numbers.  Then an edge p -> q closes
// popc(members of p & neighbours of q) triangles: those in which q is the
// middle and those in which it is the highest vertex, so that is q's credit,
// and half a row's sum is p's.  The pairs of core members are not among them
// (their lists are not looked up).  Shared-memory wavefronts bound it, so the
// table is a twentieth full -- a look-up that finds nothing mostly ends at its
// first slot -- and its bytes are the numbers themselves (RGG 4M: 402 us, 87%
// of the wavefront slots; per-row merges of sorted lists, 8 of 32 lanes busy,
// took 863.  R-MAT 22's short rows: 2160 us, at 1024 slots 2433).
template <bool PV, bool BATCH, typename Pos>
__device__ __forceinline__ void
tile_rows(const Data &w, long long u0, const VInfo &vi, int g, bool act, TileSmem<Pos> &smem,
          unsigned long long &tri)
{
    TileData<Pos> &sm = smem.tile;
    unsigned char *const slot = smem.slot;
    constexpr int kPer = 4;
    constexpr unsigned int kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned int below = (1u << lane) - 1u, upto = below | (1u << lane);
    constexpr unsigned int kMask = kTileSlots - 1;
    constexpr int kLog = ilog2(kTileSlots);
    // the rows that take part, in the first lanes
    const unsigned int acts = __ballot_sync(kAll, act);
    const int rows = __popc(acts);
    if (rows == 0) return;
    __syncwarp();
    if (act) sm.from[__popc(acts & below)] = (unsigned char)lane;
    __syncwarp();
    const int src = lane < rows ? sm.from[lane] : 0;
    int fd = __shfl_sync(kAll, vi.fdeg, src);
    if (lane >= rows) fd = 0;
    const int incl = warp_incl_scan(fd), excl = incl - fd;
    const int total = __shfl_sync(kAll, incl, 31);
    const Pos start = __shfl_sync(kAll, (Pos)vi.fbeg, src) - (Pos)excl;
    const int gr = BATCH ? __shfl_sync(kAll, g, src) : 0;
    for (int base = 0; base < total;) {
        // rows r0 .. r1 - 1, r1 <= r2: one graph (core members are positions in it)
        const int r0 = __popc(__ballot_sync(kAll, lane < rows && incl <= base));
        int stop = total;
        long long v0 = 0;
        const GraphRec *rec = w.recs;
        if (BATCH) {
            const int gf = __shfl_sync(kAll, gr, r0);
            const unsigned int other =
                __ballot_sync(kAll, lane < rows && lane > r0 && gr != gf);
            const int at = __shfl_sync(kAll, excl, other ? __ffs(other) - 1 : 0);
            if (other) stop = at;
            rec += gf;
            v0 = rec->v0;
        }
        const Lists ls = lists_of<BATCH>(w, rec);
        stop = min(stop - base, kTileEdges);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < kTileWords; ++k) {
#pragma unroll
            for (int j = 0; j < kTileIds / 32; ++j) sm.adj[k][j * 32 + lane] = 0;
            sm.begins[k * 32 + lane] = 0;
            sm.rowbits[k][lane] = 0;
        }
        __syncwarp();
        // number the members, 32 edges at a time while there is room
        int n = 0, seen = 0, row = r0 - 1;
        for (; seen < stop && n <= kTileIds - 32; seen += 32) {
            const int e = seen + lane, b = excl - base - seen;
            const unsigned int heads =
                __reduce_or_sync(kAll, lane < rows && b >= 0 && b < 32 ? 1u << b : 0u);
            const int i = row + __popc(heads & upto);
            row += __popc(heads);
            const Pos f = __shfl_sync(kAll, start, i);
            bool todo = e < stop;
            const int m = todo ? ls.base[f + (Pos)(base + e)] : 0;
            unsigned int h = hash_slot(m, kLog);
            int id = 0;
            while (__any_sync(kAll, todo)) {
                const int x = todo ? slot[h] : 0;
                bool mine = false;
                __syncwarp();                     // all have read before any claims
                if (todo) {
                    if (x == kNoId) {
                        slot[h] = (unsigned char)(kClaimed | lane);
                        mine = true;
                    } else if (sm.member[x] == m) {
                        id = x;
                        todo = false;
                    } else {
                        h = (h + 1) & kMask;
                    }
                }
                __syncwarp();
                // of the lanes that claim a slot one has it, those with the
                // same member share its number, the others go on
                const int by = mine ? slot[h] & 31 : lane;
                const bool won = mine && by == lane;
                const unsigned int wm = __ballot_sync(kAll, won);
                if (wm == 0) continue;
                if (won) id = n + __popc(wm & below);
                const int mb = __shfl_sync(kAll, m, by), ib = __shfl_sync(kAll, id, by);
                if (mine) {
                    if (mb == m) {
                        id = ib;
                        todo = false;
                    } else {
                        h = (h + 1) & kMask;
                    }
                }
                if (won) {
                    slot[h] = (unsigned char)id;
                    sm.member[id] = m;
                }
                n += __popc(wm);
                __syncwarp();
            }
            if (e < stop) {
                sm.edge[e] = (unsigned short)(id | i << 8);
                atomicOr(&sm.rowbits[id >> 5][i], 1u << (id & 31));
            }
        }
        seen = min(seen, stop);
        __syncwarp();
        // whole rows only: the edges of a cut row come again in the next tile
        const int r1 = __popc(__ballot_sync(kAll, lane < rows && incl - base <= seen));
        const int edges = __shfl_sync(kAll, incl, r1 - 1) - base;
        // y is a list element of number id
        auto look = [&](int y, auto &&owner) {
            unsigned int h = hash_slot(y, kLog);
            int x = slot[h];
            while (x != kNoId) {
                if (sm.member[x] == y) {
                    const int id = owner();
                    atomicOr(&sm.adj[id >> 5][x], 1u << (id & 31));
                    break;
                }
                h = (h + 1) & kMask;
                x = slot[h];
            }
        };
        // the lists of the members of the whole rows: lay out the stream
        int qlen[kTileWords];
        Pos qfb[kTileWords];
#pragma unroll
        for (int k = 0; k < kTileWords; ++k) {
            const unsigned int used =
                __reduce_or_sync(kAll, lane < r1 ? sm.rowbits[k][lane] : 0u);
            const int x = (used >> lane) & 1u ? sm.member[k * 32 + lane] : -1;
            qlen[k] = 0;
            qfb[k] = 0;
            if (x >= 0) {
                const VInfo q = w.vinfo[x + ls.shift];
                qlen[k] = q.fdeg;
                qfb[k] = (Pos)q.fbeg;
            }
        }
        int lists = 0, elements = 0;
#pragma unroll
        for (int k = 0; k < kTileWords; ++k) {
            const int len = qlen[k] <= kTileLong ? qlen[k] : 0;
            const int li = warp_incl_scan(len), le = elements + li - len;
            const unsigned int have = __ballot_sync(kAll, len > 0);
            if (len > 0) {
                const int o = lists + __popc(have & below);
                sm.start[o] = qfb[k] - (Pos)le;
                sm.owner[o] = (unsigned char)(k * 32 + lane);
                atomicOr(&sm.begins[le >> 5], 1u << (le & 31));
            }
            lists += __popc(have);
            elements += __shfl_sync(kAll, li, 31);
        }
        __syncwarp();
        // look its elements up, 128 at a time
        int o0 = -1;                              // lists begun before this step
        for (int f0 = 0; f0 < elements; f0 += 32 * kPer) {
            int y[kPer], o[kPer];
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int f = f0 + 32 * j + lane;
                const unsigned int word = f0 + 32 * j < elements ? sm.begins[(f0 >> 5) + j] : 0u;
                o[j] = o0 + __popc(word & upto);
                o0 += __popc(word);
                y[j] = f < elements ? ls.base[sm.start[o[j]] + (Pos)f] : kNoProbe;
            }
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                if (f0 + 32 * j >= elements) break;
                look(y[j], [&] { return (int)sm.owner[o[j]]; });
            }
        }
        // the long lists, one by one
#pragma unroll
        for (int k = 0; k < kTileWords; ++k) {
            unsigned int longs = __ballot_sync(kAll, qlen[k] > kTileLong);
            while (longs) {
                const int q = __ffs(longs) - 1;
                longs &= longs - 1;
                const int *list = ls.base + (long long)__shfl_sync(kAll, qfb[k], q);
                const int ql = __shfl_sync(kAll, qlen[k], q);
                for (int j = lane; j < ql; j += 64) {
                    const int y0 = list[j];
                    const int y1 = j + 32 < ql ? list[j + 32] : kNoProbe;
                    look(y0, [&] { return k * 32 + q; });
                    if (y1 != kNoProbe) look(y1, [&] { return k * 32 + q; });
                }
                __syncwarp();
            }
        }
        __syncwarp();
        // symmetric: with the transposed blocks
        const Transposer tr(lane);
        unsigned int block[kTileWords][kTileWords];
#pragma unroll
        for (int k = 0; k < kTileWords; ++k)
#pragma unroll
            for (int j = 0; j < kTileWords; ++j) block[k][j] = sm.adj[k][j * 32 + lane];
#pragma unroll
        for (int k = 0; k < kTileWords; ++k) {
#pragma unroll
            for (int j = 0; j < kTileWords; ++j)
                sm.adj[k][j * 32 + lane] = block[k][j] | tr(block[j][k]);
            if (PV) sm.credit[k * 32 + lane] = 0;
        }
        __syncwarp();
        // count
        unsigned int sum = 0;
        for (int e0 = 0; e0 < edges; e0 += 32) {
            const int e = e0 + lane;
            unsigned int c = 0;
            if (e < edges) {
                const int id = sm.edge[e] & 0xff, r = sm.edge[e] >> 8;
#pragma unroll
                for (int k = 0; k < kTileWords; ++k)
                    c += __popc(sm.rowbits[k][r] & sm.adj[k][id]);
                if (PV && c) atomicAdd(&sm.credit[id], c);
            }
            if (PV) {
                // a row's edges are consecutive: its lane takes a difference
                // of prefix sums
                const int ps = warp_incl_scan((int)c);
                const int lo = max(excl - base - e0, 0), hi = min(incl - base - e0, 32);
                const int top = __shfl_sync(kAll, ps, (hi - 1) & 31);
                const int bot = __shfl_sync(kAll, ps, (lo - 1) & 31);
                if (hi > lo) sum += (unsigned int)(top - (lo > 0 ? bot : 0));
            } else {
                sum += c;
            }
        }
        __syncwarp();
        if (PV) {
            sum >>= 1;
            if (sum) add64(&w.tacc[u0 + src], sum);
            tri += sum;
        } else {
            sum = warp_sum(sum) >> 1;
            tri += lane == 0 ? sum : 0u;
        }
        for (int id = lane; id < n; id += 32) {
            const int m = sm.member[id];
            if (PV) {
                const unsigned int c = sm.credit[id];
                if (c) credit(w, v0, ls.shift, m, c);
            }
            unsigned int h = hash_slot(m, kLog);
            while (slot[h] != id) h = (h + 1) & kMask;
            slot[h] = (unsigned char)kNoId;
        }
        base += edges;
    }
}

// Rows of a graph with signatures.  A pair (q, s) of a row's members, q < s,
// is an edge only if q's signature has s's bits.  W lanes per row, a member s
// each: the members' signatures are put side by side, and a lane reads its word
// of each in turn -- a warp's reads lie in eight neighbouring banks, one
// wavefront per step.  Pairs that pass are queued and searched for 32 at a time.
// Instruction issue bounds it (70%): ER 900K of mean degree 30 takes 247 us,
// tiles of the same rows 558.
template <bool PV, bool BATCH, typename Pos>
struct SignedRows {
    const Data &w;
    SignedSmem &sm;
    const long long u0;
    const VInfo &vi;
    const int g, lane;
    int queued;
    unsigned long long tri;

    // the last n (at most 32) queued pairs: s looked for in q's list
    __device__ __forceinline__ void search(int n)
    {
        __syncwarp();
        const int at = queued - n + lane;
        const int r = lane < n ? sm.row[at] : 0;
        const int v0 = BATCH ? (int)w.recs[__shfl_sync(0xffffffffu, g, r)].v0 : 0;
        if (lane < n) {
            const int q = sm.q[at], s = sm.s[at];
            const VInfo qi = w.vinfo[q + v0];
            const int *list = w.ind + qi.fbeg;
            int lo = 0, len = qi.fdeg;
            while (len > 0) {                     // first element that is not below s
                const int half = len >> 1;
                if (list[lo + half] < s) {
                    lo += half + 1;
                    len -= half + 1;
                } else {
                    len = half;
                }
            }
            if (lo < qi.fdeg && list[lo] == s) {
                ++tri;
                if (PV) {
                    add64(&w.tacc[u0 + r], 1u);
                    add64(&w.tacc[q + v0], 1u);
                    add64(&w.tacc[s + v0], 1u);
                }
            }
        }
        queued -= n;
        __syncwarp();
    }
    // bit k of hits: the pair of member k of the row, whose members are from
    // member[0] on, and this lane's member s passed
    __device__ __forceinline__ void queue(unsigned int hits, const int *member, int s, int r)
    {
        while (true) {
            const unsigned int have = __ballot_sync(0xffffffffu, hits != 0);
            if (have == 0) return;
            if (hits) {
                const int at = queued + __popc(have & ((1u << lane) - 1u));
                sm.q[at] = member[__ffs(hits) - 1];
                sm.s[at] = s;
                sm.row[at] = (unsigned char)r;
                hits &= hits - 1;
            }
            queued += __popc(have);
            if (queued >= 32) search(32);
        }
    }
    // bit k of the result: whether signature k, k = 0 .. steps - 1, of sign has
    // y's bits (readable up to the next multiple of 8)
    __device__ __forceinline__ unsigned int column(const unsigned int *sign, int y, int steps) const
    {
        const Sign m = sign_of(y);
        const unsigned int *x = sign + m.word;
        unsigned int hb = 0;
        int i = 0;
        for (; i < steps; i += 8, x += 8 * kSigWords) {
            unsigned int v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = x[kSigWords * j];
#pragma unroll
            for (int j = 0; j < 8; ++j)           // bits missing: none has the top bit
                hb = __funnelshift_l((m.bits & ~v[j]) - 1u, hb, 1);
        }
        return i ? __brev(hb) >> (32 - i) : 0u;
    }
    // the lanes' members y of row r (in: there is one) and their signatures on
    // their way to shared memory, two lanes per signature; groups of W lanes
    // one signature apart, so that they read from banks of their own
    template <int W>
    __device__ __forceinline__ void fetch(int r, bool in, int y, int *member,
                                          unsigned int *sign) const
    {
        const GraphRec *rec = &w.recs[BATCH ? __shfl_sync(0xffffffffu, g, r & 31) : 0];
        const unsigned int at = (unsigned int)(rec->ubase / kSigWords) + (unsigned int)y;
        const unsigned int ins = __ballot_sync(0xffffffffu, in);
        member[lane] = y;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int k = 16 * j + (lane >> 1), part = 4 * (lane & 1);
            const unsigned int from = __shfl_sync(0xffffffffu, at, k);
            if ((ins >> k) & 1u)
                __pipeline_memcpy_async(sign + kSigWords * (k + k / W) + part,
                                        w.find + (long long)kSigWords * from + part, 16);
        }
        __pipeline_commit();
    }
    // 32 / W rows at a time; the signatures of the next ones and the members of
    // those after them are under way meanwhile
    template <int W>
    __device__ __forceinline__ void rows_of(unsigned int rows)
    {
        constexpr int kGroups = 32 / W;
        const int grp = lane / W, gl = lane % W, g0 = grp * W;
        struct Set {
            int r, fd, y;
        };
        auto next = [&]() -> Set {
            Set t{-1, 0, 0};
#pragma unroll
            for (int k = 0; k < kGroups; ++k) {
                if (k == grp && rows) t.r = __ffs(rows) - 1;
                rows &= rows - 1;
            }
            const long long fb = __shfl_sync(0xffffffffu, vi.fbeg, t.r & 31);
            const int fd = __shfl_sync(0xffffffffu, vi.fdeg, t.r & 31);
            if (t.r >= 0) t.fd = fd;
            if (gl < t.fd) t.y = w.ind[fb + gl];
            return t;
        };
        auto issue = [&](const Set &t, int b) {
            fetch<W>(t.r, gl < t.fd, t.y, sm.member[b], sm.sign[b]);
        };
        if (rows == 0) return;
        Set now = next(), then = next();
        __syncwarp();
        issue(now, 0);
        for (int b = 0; __any_sync(0xffffffffu, now.r >= 0); b ^= 1) {
            const Set after = next();
            issue(then, b ^ 1);
            __pipeline_wait_prior(1);
            __syncwarp();
            const int most = __reduce_max_sync(0xffffffffu, now.fd);
            const unsigned int hits =
                column(sm.sign[b] + kSigWords * (g0 + grp), now.y, most - 1);
            queue(gl < now.fd ? hits & ((1u << gl) - 1u) : 0u, sm.member[b] + g0, now.y, now.r);
            __syncwarp();
            now = then;
            then = after;
        }
        __pipeline_wait_prior(0);
    }
    // rows of 33 .. 64 members, two members s per lane
    __device__ __forceinline__ void long_rows(unsigned int rows)
    {
        unsigned int *const sign = sm.sign[0];
        while (rows) {
            const int r = __ffs(rows) - 1;
            rows &= rows - 1;
            const long long fb = __shfl_sync(0xffffffffu, vi.fbeg, r);
            const int fd = __shfl_sync(0xffffffffu, vi.fdeg, r);
            const bool in = lane + 32 < fd;
            const int y0 = w.ind[fb + lane], y1 = in ? w.ind[fb + 32 + lane] : 0;
            __syncwarp();
            fetch<32>(r, true, y0, sm.member[0], sign);
            fetch<32>(r, in, y1, sm.member[1], sign + kSigWords * 32);
            __pipeline_wait_prior(0);
            __syncwarp();
            const unsigned int below = (1u << lane) - 1u;
            queue(column(sign, y0, 31) & below, sm.member[0], y0, r);
            queue(in ? column(sign, y1, 32) : 0u, sm.member[0], y1, r);
            const unsigned int hits = column(sign + kSigWords * 32, y1, fd - 33);
            queue(in ? hits & below : 0u, sm.member[1], y1, r);
        }
    }
    __device__ __forceinline__ void all(bool act)
    {
        const unsigned int r8 = __ballot_sync(0xffffffffu, act && vi.fdeg <= 8);
        const unsigned int r16 = __ballot_sync(0xffffffffu, act && vi.fdeg > 8 && vi.fdeg <= 16);
        const unsigned int r32 = __ballot_sync(0xffffffffu, act && vi.fdeg > 16 && vi.fdeg <= 32);
        const unsigned int r64 = __ballot_sync(0xffffffffu, act && vi.fdeg > 32);
        rows_of<8>(r8);
        rows_of<16>(r16);
        rows_of<32>(r32);
        long_rows(r64);
        if (queued) search(queued);
    }
};

struct TableWarpSmem {
    int key[4 * kWarpTable];                      // kNoMember = empty
    unsigned int cnt[4 * kWarpTable];
    unsigned int bits[kWarpTable];
};

struct TableBlockSmem {
    int key[1 << kTableLog2];
    unsigned int cnt[1 << kTableLog2];
    unsigned int bits[1 << (kTableLog2 - 2)];
    int next;
    unsigned long long total;                     // a row's triangles, of all its chunks
};

// Of a row that is looked up in a bitmap: most vertices and core positions of its
// graph, most members at a time; the longest list for which the table is taken, if
// there are credits, in a graph of more than kBitFew vertices and in a smaller one.
constexpr int kBitSpan = 1 << 17, kBitMembers = 4096;
constexpr int kBitFew = 1 << 15, kBitList = 256, kBitListFew = 384;

struct BitsSmem {
    unsigned int bits[kBitSpan / 32];
    unsigned short below[kBitSpan / 32];          // members in earlier words
    unsigned int cnt[kBitMembers];
    unsigned int wsum[kThreads / 32];
    int next;
    unsigned long long total;
    WideClaim claim;
};

// Whether a row of a call with the bitmap kernel is that kernel's.
template <bool PV, bool BATCH>
__device__ __forceinline__ bool in_bitmap(const Data &w, const VInfo &vi, const GraphRec *rec)
{
    const long long span = (BATCH ? (long long)rec->nv : w.n) + rec->core;
    return w.bitmaps && span <= kBitSpan &&
           vi.fdeg > (!PV ? kWarpTable : span > kBitFew ? kBitList : kBitListFew);
}

template <typename Pos>
struct ListSmem {
    union {
        TableWarpSmem warp[kThreads / 32];
        TableBlockSmem block;
        TileSmem<Pos> tile[kThreads / 32];
    };
    WideClaim claim;
};

// Shared-memory table of a row's members: linear probing, a counter per slot,
// and eight bits per slot of which a member sets the one that it hashes to.
// Most look-ups find nothing; of 32 some always met a slot that was taken, and
// the warp walked on for them.  With the bits one in 30 does.
struct MemberTable {
    int *key;
    unsigned int *cnt, *bits;
    int lg;

    // all slots empty, by the lanes or threads `id` of `count`
    template <bool PV>
    __device__ __forceinline__ void clear(int id, int count) const
    {
        const int slots = 1 << lg;
        for (int k = id; k < slots; k += count) {
            key[k] = kNoMember;
            if (PV) cnt[k] = 0;
        }
        for (int k = id; k < slots / 4; k += count) bits[k] = 0;
    }
    __device__ __forceinline__ void insert(int m) const
    {
        const unsigned int mask = (1u << lg) - 1u, b = hash_slot(m, lg + 3);
        atomicOr(&bits[b >> 5], 1u << (b & 31));
        unsigned int s = b >> 3;
        while (atomicCAS(&key[s], kNoMember, m) != kNoMember) s = (s + 1) & mask;
    }
    __device__ __forceinline__ int find(int x) const
    {
        const unsigned int mask = (1u << lg) - 1u, b = hash_slot(x, lg + 3);
        if (!((bits[b >> 5] >> (b & 31)) & 1u)) return -1;
        unsigned int s = b >> 3;
        int k = key[s];
        while (k != x && k != kNoMember) {
            s = (s + 1) & mask;
            k = key[s];
        }
        return k == x ? (int)s : -1;
    }
};

// Shared-memory bitmap of a row's members over all that its graph's lists can
// name, vertices and core positions; a member's counter is the number of
// members before it.  base: what a list calls the graph's first vertex.
template <bool PV>
struct MemberBits {
    const unsigned int *bits;
    const unsigned short *below;
    unsigned int *cnt;
    int base, nv;
    unsigned int span;

    __device__ __forceinline__ unsigned int index(int m) const
    {
        return m >= 0 ? (unsigned int)(m - base) : (unsigned int)nv + (unsigned int)~m;
    }
    __device__ __forceinline__ int find(int x) const
    {
        const unsigned int i = index(x), b = i & 31;
        if (i >= span) return -1;
        const unsigned int word = bits[i >> 5];
        if (!((word >> b) & 1u)) return -1;
        return PV ? below[i >> 5] + __popc(word & ((1u << b) - 1u)) : 0;
    }
};

// The lists of the members of list[k .. k + 32) that are not core, looked up
// by the warp: list by list where they are long, 128 elements at a time, up to
// the first above `last` (the row's highest member if lists are ascending), else
// as one stream (finding each element's list costs as much as looking it up,
// but short lists one by one would wait for memory one by one).  Returns this
// lane's member's hits.
template <bool PV, typename Pos, class Table>
__device__ __forceinline__ unsigned int probe_members(const Data &w, const Lists &ls,
                                                      const int *list, int k, int n, int last,
                                                      const Table &tab)
{
    constexpr int kPer = 4;
    const int lane = threadIdx.x & 31;
    const int m = k + lane < n ? list[k + lane] : kNoMember;
    int len = 0;
    Pos qf = 0;
    if (m >= 0) {
        const VInfo q = w.vinfo[m + ls.shift];
        len = q.fdeg;
        qf = (Pos)q.fbeg;
    }
    const int incl = warp_incl_scan(len), excl = incl - len;
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    unsigned int lists = __ballot_sync(0xffffffffu, len > 0);
    unsigned int cq = 0;
    if (total >= 64 * __popc(lists)) {
        while (lists) {
            const int src = __ffs(lists) - 1;
            lists &= lists - 1;
            const int *ql = ls.base + __shfl_sync(0xffffffffu, qf, src);
            const int n = __shfl_sync(0xffffffffu, len, src);
            unsigned int c = 0;
            for (int j0 = 0; j0 < n; j0 += 32 * kPer) {
                int x[kPer];
#pragma unroll
                for (int j = 0; j < kPer; ++j)
                    x[j] = j0 + 32 * j + lane < n ? ql[j0 + 32 * j + lane] : kNoProbe;
                if (last != INT32_MAX && __shfl_sync(0xffffffffu, x[0], 0) > last) break;
#pragma unroll
                for (int j = 0; j < kPer; ++j) {
                    if (j0 + 32 * j >= n) break;
                    const int s = tab.find(x[j]);
                    if (s >= 0) {
                        ++c;
                        if (PV) atomicAdd(&tab.cnt[s], 1u);
                    }
                }
            }
            c = warp_sum(c);
            if (lane == src) cq = c;
        }
        if (PV && cq) add64(&w.tacc[m + ls.shift], cq);
        return cq;
    }
    const Pos start = qf - (Pos)excl;
    for (int f0 = 0; f0 < total; f0 += 32 * kPer) {
        int x[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int f = f0 + 32 * j + lane;
            const Pos at = __shfl_sync(0xffffffffu, start, warp_corank(incl, f));
            x[j] = f < total ? ls.base[at + (Pos)f] : kNoProbe;
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int s = tab.find(x[j]);
            const unsigned int hm = __ballot_sync(0xffffffffu, s >= 0);
            if (PV && s >= 0) atomicAdd(&tab.cnt[s], 1u);
            cq += __popc(hm & lane_range(excl - f0 - 32 * j, incl - f0 - 32 * j));
        }
    }
    if (PV && cq) add64(&w.tacc[m + ls.shift], cq);
    return cq;
}

// A wide row of at most kWarpTable members by a warp.
template <bool PV, bool BATCH, typename Pos>
__device__ __forceinline__ void table_warp_row(const Data &w, int v, const VInfo &vi,
                                               const GraphRec *rec, TableWarpSmem &sm,
                                               unsigned long long &tri)
{
    const int lane = threadIdx.x & 31;
    const Lists ls = lists_of<BATCH>(w, rec);
    const long long v0 = BATCH ? rec->v0 : 0;
    const int *list = ls.base + vi.fbeg;
    const MemberTable tab{sm.key, sm.cnt, sm.bits, max(ceil_log2(4 * (long long)vi.fdeg), 5)};
    const int slots = 1 << tab.lg;
    __syncwarp();
    tab.clear<PV>(lane, 32);
    __syncwarp();
    // all lanes make the same steps: after a loop that each leaves by itself the
    // compiler ran all that follows for them apart where only the global count
    // was asked for (ER 200K of mean degree 100: 2858 us, 1008 so; with counts 1097)
    for (int k0 = 0; k0 < vi.fdeg; k0 += 32) {
        if (k0 + lane < vi.fdeg) tab.insert(list[k0 + lane]);
        __syncwarp();
    }
    unsigned int mine = 0;
    for (int k = 0; k < vi.fdeg; k += 32) mine += probe_members<PV, Pos>(w, ls, list, k, vi.fdeg, INT32_MAX, tab);
    mine = warp_sum(mine);
    __syncwarp();
    if (mine) {
        if (PV) {
            for (int k = lane; k < slots; k += 32)
                if (sm.cnt[k]) credit(w, v0, ls.shift, sm.key[k], sm.cnt[k]);
            if (lane == 0) add64(&w.tacc[v], mine);
        }
        tri += lane == 0 ? mine : 0u;
    }
}

// A longer one by the block, at most kMemberChunk members in the table at a
// time (a quarter full at most).  A row of f members has up to f (f - 1) / 2
// triangles, more than 32 bits hold from f = 92,683 on, so its total is 64 bits
// wide.  What a warp finds in one chunk is at most kMemberChunk per list, and f
// stays below 2^22 (a degree that no one of f others is below, or that is at most
// twice the mean and 16, takes f * f / 2 entries, 2^43): 32 bits hold it, and a
// member's count, at most f, as well.
template <bool PV, bool BATCH, typename Pos>
__device__ void table_block_row(const Data &w, int v, const VInfo &vi, const GraphRec *rec,
                                TableBlockSmem &sm, unsigned long long &tri)
{
    const int lane = threadIdx.x & 31;
    const Lists ls = lists_of<BATCH>(w, rec);
    const long long v0 = BATCH ? rec->v0 : 0;
    const int *list = ls.base + vi.fbeg;
    __syncthreads();
    if (threadIdx.x == 0) sm.total = 0;
    // members whose lists a warp takes at a time: four shares per warp at
    // least (R-MAT 22, wide rows: 5140 us at 32 members always, 4726 so)
    const int per = max(4, min(32, vi.fdeg / (4 * kThreads / 32)));
    for (int c0 = 0; c0 < vi.fdeg; c0 += kMemberChunk) {
        const int nm = min(vi.fdeg - c0, kMemberChunk);
        const MemberTable tab{sm.key, sm.cnt, sm.bits,
                              min(max(ceil_log2(8 * (long long)nm), 6), kTableLog2)};
        const int slots = 1 << tab.lg;
        tab.clear<PV>(threadIdx.x, kThreads);
        if (threadIdx.x == 0) sm.next = 0;
        __syncthreads();
        for (int k = threadIdx.x; k < nm; k += kThreads) tab.insert(list[c0 + k]);
        __syncthreads();
        unsigned int mine = 0;
        while (true) {
            int k = 0;
            if (lane == 0) k = atomicAdd(&sm.next, per);
            k = __shfl_sync(0xffffffffu, k, 0);
            if (k >= vi.fdeg) break;
            mine += probe_members<PV, Pos>(w, ls, list, k, min(k + per, vi.fdeg), INT32_MAX, tab);
        }
        __syncthreads();
        if (PV)
            for (int k = threadIdx.x; k < slots; k += kThreads)
                if (sm.cnt[k]) credit(w, v0, ls.shift, sm.key[k], sm.cnt[k]);
        const unsigned int ws = warp_sum(mine);
        if (lane == 0 && ws) atomicAdd(&sm.total, (unsigned long long)ws);
        __syncthreads();
    }
    if (threadIdx.x == 0 && sm.total) {
        if (PV) atomicAdd(&w.tacc[v], sm.total);
        tri += sm.total;
    }
}

// A longer row of a graph of at most kBitSpan vertices and core positions, in a
// bitmap of all of them: kBitMembers members at a time, so mostly in one pass over
// the lists where the table makes one per kMemberChunk, and a hit needs no key.
// Instruction issue bounds it (77%).  Sums as in table_block_row.  ER 40K of mean degree 2,000 42 ms (table 91; binary
// search of degree-sorted lists, which the tables replaced, 39), ring of 40K with
// 1,000 neighbours each, in no order of ids, 11.5 (16.9; 11.3).  Where the lines
// are, with credits: from 257 members on ER 40K of 500 takes 3.14 ms, RGG 100K of
// 500 10.3, from 385 on 3.27 and 11.1; but 200 graphs ER 5K of 300 40.7 and 37.5,
// R-MAT 14 of 256 0.285 from 129 on and 0.255.  Without credits from the first row
// on that a block takes: ER 40K of 500 2.63 (table 3.11), RGG 100K 7.5 (10.1).
template <bool PV, bool BATCH, typename Pos>
__device__ void bits_block_row(const Data &w, int v, const VInfo &vi, const GraphRec *rec,
                               BitsSmem &sm, unsigned long long &tri)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Lists ls = lists_of<BATCH>(w, rec);
    const long long v0 = BATCH ? rec->v0 : 0;
    const int *list = ls.base + vi.fbeg;
    const int last = rec->uniform ? list[vi.fdeg - 1] : INT32_MAX;
    const int nv = BATCH ? rec->nv : (int)w.n, span = nv + rec->core;
    const MemberBits<PV> tab{sm.bits, sm.below, sm.cnt, BATCH ? (int)v0 - ls.shift : 0, nv,
                             (unsigned int)span};
    const int words = (span + 31) >> 5, each = div_up(words, kThreads);
    const int per = max(4, min(32, vi.fdeg / (4 * kThreads / 32)));
    __syncthreads();
    if (threadIdx.x == 0) sm.total = 0;
    for (int c0 = 0; c0 < vi.fdeg; c0 += kBitMembers) {
        const int nm = min(vi.fdeg - c0, kBitMembers);
        for (int k = threadIdx.x; k < words; k += kThreads) sm.bits[k] = 0;
        if (PV)
            for (int k = threadIdx.x; k < nm; k += kThreads) sm.cnt[k] = 0;
        if (threadIdx.x == 0) sm.next = 0;
        __syncthreads();
        for (int k = threadIdx.x; k < nm; k += kThreads) {
            const unsigned int i = tab.index(list[c0 + k]);
            if (i < tab.span) atomicOr(&sm.bits[i >> 5], 1u << (i & 31));
        }
        __syncthreads();
        if (PV) {
            const int w0 = (int)threadIdx.x * each;
            int sum = 0;
            for (int j = 0; j < each; ++j)
                if (w0 + j < words) sum += __popc(sm.bits[w0 + j]);
            const int incl = warp_incl_scan(sum);
            if (lane == 31) sm.wsum[warp] = (unsigned int)incl;
            __syncthreads();
            int first = incl - sum;
            for (int i = 0; i < warp; ++i) first += (int)sm.wsum[i];
            for (int j = 0; j < each; ++j)
                if (w0 + j < words) {
                    sm.below[w0 + j] = (unsigned short)first;
                    first += __popc(sm.bits[w0 + j]);
                }
            __syncthreads();
        }
        unsigned int mine = 0;
        while (true) {
            int k = 0;
            if (lane == 0) k = atomicAdd(&sm.next, per);
            k = __shfl_sync(0xffffffffu, k, 0);
            if (k >= vi.fdeg) break;
            mine += probe_members<PV, Pos>(w, ls, list, k, min(k + per, vi.fdeg), last, tab);
        }
        __syncthreads();
        if (PV)
            for (int k = threadIdx.x; k < nm; k += kThreads) {
                const int m = list[c0 + k];
                const int s = tab.find(m);
                const unsigned int c = s >= 0 ? sm.cnt[s] : 0u;
                if (c) credit(w, v0, ls.shift, m, c);
            }
        const unsigned int ws = warp_sum(mine);
        if (lane == 0 && ws) atomicAdd(&sm.total, (unsigned long long)ws);
        __syncthreads();
    }
    if (threadIdx.x == 0 && sm.total) {
        if (PV) atomicAdd(&w.tacc[v], sm.total);
        tri += sm.total;
    }
}

template <bool PV, bool BATCH, typename Pos>
__device__ __forceinline__ void table_wide_rows(const Data &w, ListSmem<Pos> &sm,
                                                unsigned long long &tri)
{
    // a member outside the core, and one more (core rows have none)
    wide_rows(
        w, sm.claim, first_block(w.n, gridDim.x / 4), &w.ctr->table_long_next, &w.ctr->table_wide_next, kWarpTable,
        [](const VInfo &vi) { return vi.fdeg >= 2 && vi.fdeg > (vi.dk & INT32_MAX); },
        [&](int v, const VInfo &vi) {
            const GraphRec *rec = &w.recs[BATCH ? w.gid[v] : 0];
            if (!in_bitmap<PV, BATCH>(w, vi, rec))
                table_block_row<PV, BATCH, Pos>(w, v, vi, rec, sm.block, tri);
        },
        [&](int v, const VInfo &vi) {
            table_warp_row<PV, BATCH, Pos>(w, v, vi, &w.recs[BATCH ? w.gid[v] : 0],
                                      sm.warp[threadIdx.x >> 5], tri);
        });
}

// Rows u0 .. u0 + batch - 1 that are short, those of graphs with signatures
// (SIGN) and the others (TILE).
template <bool PV, bool BATCH, bool TILE, bool SIGN, typename Pos>
__device__ __forceinline__ void list_rows(const Data &w, long long u0, int batch,
                                          TileSmem<Pos> &sm, unsigned long long &tri)
{
    const int lane = threadIdx.x & 31;
    VInfo vi{0, 0, 0};
    int g = 0;
    if (lane < batch && u0 + lane < w.n) {
        vi = w.vinfo[u0 + lane];
        if (BATCH) g = w.gid[u0 + lane];
    }
    // not a wide row, at least one member outside the core and one more
    const bool act = vi.dk >= 0 && vi.fdeg >= 2 && vi.fdeg > vi.dk;
    const bool sign = SIGN && act && (!TILE || w.recs[g].uniform == kSigned);
    if (SIGN && __any_sync(0xffffffffu, sign)) {
        SignedRows<PV, BATCH, Pos> rows{w, sm.sign, u0, vi, g, lane, 0, 0};
        rows.all(sign);
        tri += rows.tri;
    }
    if (TILE) tile_rows<PV, BATCH, Pos>(w, u0, vi, g, act && !sign, sm, tri);
}

// ================================================================== kernels

// Warps take `batch` consecutive rows at a time: their own share first, then
// from a queue.
template <class Rows>
__device__ __forceinline__ void warp_batches(unsigned long long *queue, long long n, int batch,
                                             const Rows &rows)
{
    const long long all = (long long)gridDim.x * (kThreads / 32) * batch;
    const long long block = first_block(n, gridDim.x / 2);
    long long u0 = (block * (kThreads / 32) + (threadIdx.x >> 5)) * batch;
    while (u0 < n) {
        rows(u0);
        if (all >= n) break;
        if ((threadIdx.x & 31) == 0)
            u0 = all + (long long)atomicAdd(queue, (unsigned long long)batch);
        u0 = __shfl_sync(0xffffffffu, u0, 0);
    }
}

__device__ __forceinline__ void add_triangles(Counters *ctr, unsigned long long tri)
{
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) tri += __shfl_down_sync(0xffffffffu, tri, d);
    if ((threadIdx.x & 31) == 0 && tri) atomicAdd(&ctr->tri_total, tri);
}

// Whether sparse_core_kernel takes the short rows.
__device__ __forceinline__ bool by_pairs(const Data &w)
{
    return w.sparse && w.recs[0].uniform == 1;
}

// All short rows: rows(u0, ..) of list_rows, then also(u0).  A single graph is
// all tiles or all signatures, each in a loop with registers of its own.
template <bool PV, bool BATCH, typename Pos, class Also>
__device__ __forceinline__ void list_short_rows(const Data &w, int batch, TileSmem<Pos> &sm,
                                                unsigned long long &tri, const Also &also)
{
    unsigned long long *queue = &w.ctr->list_short_next;
    if (!BATCH && by_pairs(w)) return;            // no core either
    if (!BATCH && w.recs[0].uniform == kSigned) {
        warp_batches(queue, w.n, batch, [&](long long u0) {
            list_rows<PV, BATCH, false, true, Pos>(w, u0, batch, sm, tri);
        });
        return;
    }
    tile_init(sm);
    warp_batches(queue, w.n, batch, [&](long long u0) {
        list_rows<PV, BATCH, true, BATCH, Pos>(w, u0, batch, sm, tri);
        also(u0);
    });
}

template <bool BATCH>
__device__ __forceinline__ bool has_core(const Data &w)
{
    return (BATCH ? (long long)w.ctr->u_words : (long long)w.recs[0].core) != 0;
}

template <bool PV, bool BATCH>
__global__ void __launch_bounds__(kThreads, 4)
core_kernel(const Data w, bool do_wide, bool do_short, int batch)
{
    __shared__ CoreSmem sm;
    if (gated(w) || !has_core<BATCH>(w)) return;
    unsigned long long tri = 0;
    if (do_wide) core_wide_rows<PV, BATCH>(w, sm, tri);
    if (do_short)
        warp_batches(&w.ctr->core_short_next, w.n, batch, [&](long long u0) {
            core_short_rows<PV, BATCH>(w, u0, batch, tri);
        });
    add_triangles(w.ctr, tri);
}

// Short rows of a sparse uniform graph (RowConfig::sparse): 32 rows per warp, their
// pairs (q, s) of members, q < s, as one stream, s looked for in q's list.  A tile
// costs the same however few edges its rows have; here rows of one member cost a
// load, the next rows' on its way.  Waits for lists bound it, then issue (54%) at 32
// warps per SM.  Grid of 2000 x 2000: tiles 173 us, 61 here; path of 8 M vertices
// 176 and 47.
template <bool PV>
__device__ __forceinline__ void pair_rows(const Data &w, unsigned long long &tri)
{
    constexpr int kPer = 2;                       // pairs in flight per lane
    const int lane = threadIdx.x & 31;
    const long long step = (long long)gridDim.x * kThreads;
    long long u0 = (long long)blockIdx.x * kThreads + (threadIdx.x & ~31);
    auto row = [&](long long u) {
        return u + lane < w.n ? w.vinfo[u + lane] : VInfo{0, 0, 0};
    };
    for (VInfo vi = row(u0); u0 < w.n; u0 += step) {
        const VInfo next = row(u0 + step);
        const int n = vi.dk >= 0 ? vi.fdeg * (vi.fdeg - 1) / 2 : 0;     // wide rows: none
        const int incl = warp_incl_scan(n), excl = incl - n;
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        for (int f0 = 0; f0 < total; f0 += 32 * kPer) {
            int r[kPer], q[kPer], s[kPer];
            VInfo qi[kPer];
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int f = f0 + 32 * j + lane;
                r[j] = warp_corank(incl, f);
                const int p = f - __shfl_sync(0xffffffffu, excl, r[j]);
                const int *list = w.ind + __shfl_sync(0xffffffffu, vi.fbeg, r[j]);
                q[j] = s[j] = -1;
                if (f < total) {
                    int b = (int)((sqrtf(8.0f * (float)p + 1.0f) + 1.0f) * 0.5f);
                    while (b * (b - 1) / 2 > p) --b;
                    while (b * (b + 1) / 2 <= p) ++b;
                    q[j] = list[p - b * (b - 1) / 2];
                    s[j] = list[b];
                }
            }
#pragma unroll
            for (int j = 0; j < kPer; ++j)
                qi[j] = q[j] >= 0 ? w.vinfo[q[j]] : VInfo{0, 0, 0};
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int *list = w.ind + qi[j].fbeg;
                int lo = 0, len = qi[j].fdeg;
                while (len > 0) {                 // first element that is not below s
                    const int half = len >> 1;
                    if (list[lo + half] < s[j]) {
                        lo += half + 1;
                        len -= half + 1;
                    } else {
                        len = half;
                    }
                }
                if (lo < qi[j].fdeg && list[lo] == s[j]) {
                    ++tri;
                    if (PV) {
                        add64(&w.tacc[u0 + r[j]], 1u);
                        add64(&w.tacc[q[j]], 1u);
                        add64(&w.tacc[s[j]], 1u);
                    }
                }
                __syncwarp();
            }
        }
        vi = next;
    }
}

// core_kernel of a sparse graph: pairs of short rows if the graph is uniform, core
// pairs if not.  Pairs in a kernel of their own took 47 and 37 us, but a launch more
// than gtc_count_launches has always said for such a graph.
template <bool PV>
__global__ void __launch_bounds__(kThreads, 4)
sparse_core_kernel(const Data w, bool do_wide, bool do_short, int batch)
{
    __shared__ CoreSmem sm;
    if (gated(w)) return;
    unsigned long long tri = 0;
    if (by_pairs(w)) {
        if (do_short) pair_rows<PV>(w, tri);
    } else if (has_core<false>(w)) {
        if (do_wide) core_wide_rows<PV, false>(w, sm, tri);
        if (do_short)
            warp_batches(&w.ctr->core_short_next, w.n, batch, [&](long long u0) {
                core_short_rows<PV, false>(w, u0, batch, tri);
            });
    }
    add_triangles(w.ctr, tri);
}

template <bool PV, bool BATCH, typename Pos>
__global__ void __launch_bounds__(kThreads, 5)
list_kernel(const Data w, bool do_wide, bool do_short, int batch)
{
    extern __shared__ __align__(16) unsigned char smem[];
    if (gated(w)) return;
    ListSmem<Pos> &sm = *reinterpret_cast<ListSmem<Pos> *>(smem);
    unsigned long long tri = 0;
    if (do_wide && w.ctr->wide_rows > 0) {
        table_wide_rows<PV, BATCH, Pos>(w, sm, tri);
        __syncthreads();
    }
    if (do_short)
        list_short_rows<PV, BATCH, Pos>(w, batch, sm.tile[threadIdx.x >> 5], tri,
                                        [](long long) {});
    add_triangles(w.ctr, tri);
}

// Wide rows that a bitmap holds.  A kernel of its own, launched where rows are
// long (RowConfig::dense): as a part of list_kernel it cost R-MAT 22 0.8% and a
// ring of 400K with 100 neighbours each 3%, in registers.
template <bool PV, bool BATCH, typename Pos>
__global__ void __launch_bounds__(kThreads, 5)
bitmap_kernel(const Data w)
{
    __shared__ BitsSmem sm;
    if (gated(w)) return;
    unsigned long long tri = 0;
    wide_block_rows(
        w, sm.claim, blockIdx.x, &w.ctr->bitmap_next, PV ? kBitList : kWarpTable,
        [](const VInfo &vi) { return vi.fdeg > (vi.dk & INT32_MAX); },
        [&](int v, const VInfo &vi) {
            const GraphRec *rec = &w.recs[BATCH ? w.gid[v] : 0];
            if (in_bitmap<PV, BATCH>(w, vi, rec))
                bits_block_row<PV, BATCH, Pos>(w, v, vi, rec, sm, tri);
        });
    add_triangles(w.ctr, tri);
}

// Both, for small graphs, whose time is launches and latency.
template <bool PV, bool BATCH, typename Pos>
__global__ void __launch_bounds__(kThreads, 4)
count_kernel(const Data w, int batch)
{
    extern __shared__ __align__(16) unsigned char smem[];
    if (gated(w)) return;
    union Smem {
        ListSmem<Pos> list;
        CoreSmem core;
    };
    Smem &sm = *reinterpret_cast<Smem *>(smem);
    unsigned long long tri = 0;
    const bool core = has_core<BATCH>(w);
    if (w.ctr->wide_rows > 0) {
        if (core) core_wide_rows<PV, BATCH>(w, sm.core, tri);
        __syncthreads();
        table_wide_rows<PV, BATCH, Pos>(w, sm.list, tri);
        __syncthreads();
    }
    list_short_rows<PV, BATCH, Pos>(w, batch, sm.list.tile[threadIdx.x >> 5], tri,
                                    [&](long long u0) {
                                        if (core) core_short_rows<PV, BATCH>(w, u0, batch, tri);
                                    });
    add_triangles(w.ctr, tri);
}

// ================================================================ epilogue

__device__ __forceinline__ void write_global(const Counters *ctr, long long *global)
{
    const long long T = (long long)ctr->tri_total;
    global[0] = T;
    global[1] = 3 * T;
    global[2] = 6 * T;
}

__global__ void global_kernel(const Counters *ctr, long long *global)
{
    write_global(ctr, global);
}

// Batch in split launches: the core's credits go to their vertices.
__global__ void core_credits_kernel(const Data w)
{
    const long long rows = (long long)w.ctr->wide_rows;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += stride) {
        const int v = w.wide[i];
        const GraphRec *rec = &w.recs[w.gid[v]];
        const int k = w.key[v];
        if (k > kKeyTop - rec->core) w.tacc[v] += w.tcore[rec->v0 + kKeyTop - k];
    }
}

// r, t, lcc of every vertex; a batch's sums of t per graph; thread 0 also
// writes the global counts (nullable).
template <typename OffT, bool BATCH>
__global__ void __launch_bounds__(kThreads)
finalize_kernel(const View<OffT> w, bool credits, long long *__restrict__ r,
                long long *__restrict__ t, double *__restrict__ lcc, long long *global)
{
    const long long v = (long long)blockIdx.x * kThreads + threadIdx.x;
    if (v == 0 && global) write_global(w.ctr, global);
    unsigned long long tv = 0;
    int g = -1;
    if (v < w.n) {
        tv = w.tacc[v];
        if (BATCH) g = w.gid[v];
        if (credits) {
            const GraphRec *rec = &w.recs[BATCH ? g : 0];
            if (rec->core > 0) {
                const int k = w.key[v];
                if (k > kKeyTop - rec->core)
                    tv += w.tcore[(BATCH ? rec->v0 : 0) + kKeyTop - k];
            }
        }
        if (r) r[v] = (long long)(2 * tv);
        if (t) t[v] = (long long)tv;
        if (lcc) {
            const long long d = row_degree(w, v);
            // one IEEE division of exactly converted integers (bit-identical
            // to the host formula)
            lcc[v] = d < 2 ? 0.0 : __ddiv_rn((double)(2 * tv), (double)(d * (d - 1)));
        }
    }
    if (BATCH && w.gsum) {
        // a warp within one graph adds once
        const int g_all = __shfl_sync(0xffffffffu, g, 0);
        if (__all_sync(0xffffffffu, g == g_all || g < 0) && g_all >= 0) {
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) tv += __shfl_down_sync(0xffffffffu, tv, d);
            if ((threadIdx.x & 31) == 0 && tv) atomicAdd(&w.gsum[g_all], tv);
        } else if (g >= 0 && tv) {
            atomicAdd(&w.gsum[g], tv);
        }
    }
}

__global__ void graph_triangles_kernel(const unsigned long long *__restrict__ gsum, long long G,
                                       long long *__restrict__ graph_T)
{
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g < G) graph_T[g] = (long long)(gsum[g] / 3);
}

}  // namespace gtc
