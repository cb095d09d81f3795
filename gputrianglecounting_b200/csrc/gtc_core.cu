// gtc_core.cu -- host side of the counting pipeline: workspace layout, launch
// plan, launches.
//
// Reference operator replaced: count_all_trianglesGPU<T,bs> + kernelCall<T>
// (src/clusteringCount.cu:314-359, :415-467) and the thrust::reduce global
// sum (src/gpurun.cu:40).
#include <nvtx3/nvToolsExt.h>

#include "gtc_core.cuh"
#include "gtc_count.cuh"

namespace gtc {

namespace {

// Host-side NVTX range around the launches of one pipeline phase (header-only
// NVTX 3: a no-op unless a profiler injects itself).
struct NvtxRange {
    explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange &) = delete;
    NvtxRange &operator=(const NvtxRange &) = delete;
};

int g_sm_count[64];

int device_sm_count(int dev)
{
    if (dev < 0 || dev >= 64) return 148;
    if (!g_sm_count[dev]) {
        int v = 0;
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        g_sm_count[dev] = v > 0 ? v : 148;
    }
    return g_sm_count[dev];
}

// Blocks of a persistent kernel: every resident block, at most `work`.
template <auto Kernel>
unsigned grid_for(size_t dyn_smem, int dev, long long work)
{
    static int cache[64];                         // per kernel
    int blocks = dev >= 0 && dev < 64 ? cache[dev] : 0;
    if (!blocks) {
        if (dyn_smem > 48 * 1024)
            cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)dyn_smem);
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, Kernel, kThreads, dyn_smem);
        blocks = (per_sm < 1 ? 1 : per_sm) * device_sm_count(dev);
        if (dev >= 0 && dev < 64) cache[dev] = blocks;
    }
    return (unsigned)(work < 1 ? 1 : (work < blocks ? work : blocks));
}

inline size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// Bytes a count asks for at least: per vertex 40 (48 with counts), per entry
// 4.5, and 67 KiB; a batch adds a copy of the ids and per-graph histograms.
// The layout below fits into it with room to spare for a bit matrix, so the
// size is a contract with callers rather than a sum of today's arrays.
size_t required_bytes(long long n, long long nnz, bool per_vertex, long long graphs)
{
    size_t o = 0;
    auto take = [&](size_t bytes) { o = align256(o + bytes); };
    const size_t sn = (size_t)n, sz = (size_t)nnz;
    take(4);
    take(64);
    take(8 * 8192);
    for (int i = 0; i < 4; ++i) take(4 * sn);
    take(16 * sn);
    take(4 * (sz + 4));
    take(per_vertex ? 8 * sn : 0);
    take(8 * (size_t)(div_up<long long>(n + nnz, 2048) + 1));
    take(8 * (size_t)(div_up<long long>(nnz, 32) + 1));
    take(8 * (size_t)(n + div_up<long long>(nnz, 32) + 1));
    take(4 * (sz / 65 + 1));
    if (graphs > 0) {
        const long long buckets = graphs * 1024;
        take(8 * (size_t)(graphs + 1));
        take(4 * (sz + 1));
        take(8 * (size_t)(buckets + 1));
        take(8 * (size_t)(div_up<long long>(buckets, 8192) + 1));
        take(4 * (sn + 1));
    }
    return o;
}

}  // namespace

Plan make_plan(long long n, long long nnz, int off_bits, bool per_vertex, long long graphs)
{
    (void)off_bits;
    Plan p;
    size_t o = 0;
    auto take = [&](size_t bytes) { size_t at = o; o = align256(o + bytes); return at; };
    const long long recs = graphs > 0 ? graphs : 1;
    p.o_status = take(sizeof(unsigned int));
    p.o_counters = take(sizeof(Counters));
    p.o_hist = take(sizeof(unsigned int) * (size_t)(recs * kBuckets));
    p.o_gsum = take(sizeof(unsigned long long) * (size_t)graphs);
    // core credits: by vertex in a batch (a graph's start + position)
    const long long cores = graphs > 0 ? n : (n < kCoreMax ? n : kCoreMax);
    p.o_tcore = take(per_vertex ? sizeof(unsigned long long) * (size_t)cores : 0);
    p.o_tacc = take(per_vertex ? sizeof(unsigned long long) * (size_t)n : 0);
    p.zero_bytes = o;
    p.o_recs = take(sizeof(GraphRec) * (size_t)recs);
    p.o_key = take(sizeof(int) * (size_t)n);
    p.o_gid = take(graphs > 0 ? sizeof(int) * (size_t)n : 0);
    p.o_vinfo = take(sizeof(VInfo) * (size_t)n);
    p.o_find = take(sizeof(int) * (size_t)(nnz + 4));
    p.o_wide = take(sizeof(int) * (size_t)(n + 1));
    p.o_litem = take(sizeof(int2) * (size_t)(n + nnz / kRowChunk + 1));
    p.o_u = o;
    p.need = required_bytes(n, nnz, per_vertex, graphs);
    if (p.need < o) p.need = o;
    // bit matrix: 64 bytes per vertex (32 sqrt(n) core vertices), or all of a
    // small dense graph; a batch uses what the required size leaves, some 4
    // bytes per entry
    long long u = 64 * n;
    if (graphs > 0) {
        u = 0;
    } else {
        const long long most = n < kCoreMax ? n : kCoreMax;
        const long long full = 4ll * u_row((int)most);
        if (n <= kCoreMax && n * n <= 32 * nnz && nnz >= 64 * n && u < full) u = full;
        if (u > full) u = full;
    }
    p.bytes = align256(o + (size_t)u);
    if (p.bytes < p.need) p.bytes = p.need;
    return p;
}

RowConfig pick_row_config(long long n, long long nnz)
{
    RowConfig c;
    // Split launches are no faster anywhere that was measured (joint and split,
    // us: R-MAT 17 193 and 242, 18 396 and 429, 20 1518 and 1552, 21 3952 and
    // 4027, 22 10886 and 11040; ER 900K of mean degree 30 377 and 392; the
    // 512-graph batch 10267 and 10455).  They stay the form of large heavy graphs
    // because callers ask gtc_count_launches for the number of launches and the
    // form; from 2^18 vertices on they cost 1 to 4 percent
    c.split = n >= kSmallGraph && (double)nnz / (double)n > 24.0;
    c.sparse = n >= kSmallGraph && nnz <= 4 * n;
    c.dense = nnz >= 128 * n && !(n <= kCoreMax && n * n <= 32 * nnz);
    return c;
}

gtc_status apply_tuning(RowConfig &cfg, const gtc_tuning *tuning)
{
    if (!tuning) return GTC_OK;
    if (tuning->group && tuning->group != 4 && tuning->group != 8 && tuning->group != 16 &&
        tuning->group != 32)
        return GTC_ERR_INVALID_ARGUMENT;
    if (tuning->item_len < 0 || (tuning->item_len > 0 && tuning->item_len < 32) ||
        tuning->item_len > 32768 || (tuning->item_len & (tuning->item_len - 1)) ||
        tuning->big_chunk < 0 || (tuning->big_chunk > 0 && tuning->big_chunk < 32) ||
        tuning->big_chunk > 32768 || tuning->big_hash_max < 0 || tuning->big_hash_max > 2048 ||
        tuning->labels < 0 || tuning->labels > 2 ||
        (tuning->region != 0 && tuning->region != 2 && tuning->region != 4) ||
        tuning->rows < 0 || tuning->rows > 2 ||
        (tuning->rows == GTC_ROWS_MERGE && tuning->labels == GTC_LABELS_DEGREE_RANK))
        return GTC_ERR_INVALID_ARGUMENT;
    if (tuning->labels == GTC_LABELS_VERTEX_ID || tuning->rows == GTC_ROWS_MERGE)
        cfg.split = false;
    if (tuning->labels == GTC_LABELS_DEGREE_RANK) cfg.split = true;
    return GTC_OK;
}

int launches_per_count(const RowConfig &cfg, bool per_vertex, long long n)
{
    // split: degrees, core choice, core keys, placement of long and of short
    // rows, lists and bit matrix for each, per-vertex outputs, global counts;
    // otherwise degrees with the core choice, core keys, placement, lists and
    // bit matrix (one launch below kSmallGraph vertices), outputs; either way
    // bitmaps for a graph of long rows that they hold
    const int more = cfg.dense && n <= kBitSpan ? 1 : 0;
    if (cfg.split) return (per_vertex ? 11 : 10) + more;
    return (n >= kSmallGraph ? 6 : 5) + more;
}

namespace {

// Rows per warp batch of a persistent kernel of `blocks` blocks: 32, fewer
// where that would leave warps with less than two batches each.
int rows_per_batch(unsigned blocks, long long n)
{
    int batch = 32;
    while (batch > 2 && n < 2ll * blocks * (kThreads / 32) * batch) batch >>= 1;
    return batch;
}

template <bool PV, bool BATCH>
void launch_core(const Data &w, int dev, cudaStream_t s, bool wide, bool shrt)
{
    if (!BATCH && w.sparse) {
        constexpr auto k = sparse_core_kernel<PV>;
        const unsigned blocks = grid_for<k>(0, dev, w.n);
        k<<<blocks, kThreads, 0, s>>>(w, wide, shrt, rows_per_batch(blocks, w.n));
        return;
    }
    constexpr auto k = core_kernel<PV, BATCH>;
    const unsigned blocks = grid_for<k>(0, dev, w.n);
    k<<<blocks, kThreads, 0, s>>>(w, wide, shrt, rows_per_batch(blocks, w.n));
}

template <bool PV, bool BATCH, typename Pos>
void launch_lists(const Data &w, int dev, cudaStream_t s, bool wide, bool shrt)
{
    constexpr auto k = list_kernel<PV, BATCH, Pos>;
    const size_t smem = sizeof(ListSmem<Pos>);
    const unsigned blocks = grid_for<k>(smem, dev, w.n);
    k<<<blocks, kThreads, smem, s>>>(w, wide, shrt, rows_per_batch(blocks, w.n));
}

template <bool PV, bool BATCH, typename Pos>
void launch_both(const Data &w, int dev, cudaStream_t s)
{
    constexpr auto k = count_kernel<PV, BATCH, Pos>;
    const size_t smem = sizeof(ListSmem<Pos>) > sizeof(CoreSmem) ? sizeof(ListSmem<Pos>) : sizeof(CoreSmem);
    const unsigned blocks = grid_for<k>(smem, dev, w.n);
    k<<<blocks, kThreads, smem, s>>>(w, rows_per_batch(blocks, w.n));
}

template <typename OffT, bool BATCH, bool PV, typename Pos>
gtc_status launch(const View<OffT> &w, GraphRec lim, long long *r, long long *t, double *lcc,
                  long long *global, long long *graph_T, cudaStream_t s, const RowConfig &cfg,
                  CountTimings *timing)
{
    int dev = 0;
    cudaGetDevice(&dev);
    const long long n = w.n;
    const unsigned vb = (unsigned)div_up<long long>(n, kThreads);
    const unsigned gb = (unsigned)div_up<long long>(w.graphs, kThreads);
    const unsigned sms = (unsigned)device_sm_count(dev);
    if (timing) cudaEventRecord(timing->ev[0], s);
    {
        NvtxRange range("gtc: forward lists");
        if (BATCH && cfg.split) {
            graph_limits_kernel<<<gb, kThreads, 0, s>>>(w);
            graph_ids_kernel<<<vb, kThreads, 0, s>>>(w);
        }
        degree_kernel<OffT, BATCH><<<vb < sms * 8 ? vb : sms * 8, kThreads, 0, s>>>(
            w, lim, !cfg.split, !BATCH && !cfg.split);
        if (BATCH || cfg.split) {
            // one graph per block up to four rounds of blocks
            const long long per = min((long long)kThreads, max(1ll, w.graphs / (sms * 32)));
            const unsigned cb = BATCH ? (unsigned)div_up(w.graphs, per) : 1u;
            choose_core_kernel<OffT, BATCH><<<cb, kThreads, 0, s>>>(w, lim, !cfg.split, (int)per);
        }
        key_rows_kernel<<<n < sms * 4 * kThreads ? vb : sms * 4, kThreads, 0, s>>>(
            w, !(BATCH && cfg.split));
        if (BATCH && cfg.split) zero_bits_kernel<<<sms * 4, kThreads, 0, s>>>(w);
        constexpr auto place = place_kernel<OffT, BATCH>;
        const unsigned pb = grid_for<place>(0, dev, n);
        // rows per warp: up to 32, no more than a round needs (R-MAT 10: 9.0 us
        // at 32, 5.2 at 2; two rounds from the queue cost ER 16K 9.9 us, one 4.2)
        int batch = 2;
        while (batch < 32 && (long long)pb * (kThreads / 32) * batch < n) batch <<= 1;
        if (cfg.split) {
            place<<<pb, kThreads, 0, s>>>(w, true, false, batch);
            place<<<pb, kThreads, 0, s>>>(w, false, true, batch);
        } else {
            place<<<pb, kThreads, 0, s>>>(w, true, true, batch);
        }
    }
    if (timing) cudaEventRecord(timing->ev[1], s);
    if (w.bitmaps) {
        constexpr auto k = bitmap_kernel<PV, BATCH, Pos>;
        k<<<grid_for<k>(0, dev, n), kThreads, 0, s>>>(w);
    }
    if (cfg.split) {
        NvtxRange range("gtc: split count");
        launch_lists<PV, BATCH, Pos>(w, dev, s, true, false);
        launch_lists<PV, BATCH, Pos>(w, dev, s, false, true);
        if (timing) cudaEventRecord(timing->ev[2], s);
        launch_core<PV, BATCH>(w, dev, s, true, false);
        launch_core<PV, BATCH>(w, dev, s, false, true);
    } else if (n >= kSmallGraph) {
        NvtxRange range("gtc: count");
        launch_lists<PV, BATCH, Pos>(w, dev, s, true, true);
        if (timing) cudaEventRecord(timing->ev[2], s);
        launch_core<PV, BATCH>(w, dev, s, true, true);
    } else {
        NvtxRange range("gtc: small count");
        launch_both<PV, BATCH, Pos>(w, dev, s);
        if (timing) cudaEventRecord(timing->ev[2], s);
    }
    if (timing) cudaEventRecord(timing->ev[3], s);
    if (BATCH && cfg.split) core_credits_kernel<<<sms * 4, kThreads, 0, s>>>(w);
    const bool outputs = PV && (r || t || lcc || graph_T);
    if (outputs)
        finalize_kernel<OffT, BATCH><<<vb, kThreads, 0, s>>>(w, !(BATCH && cfg.split), r, t, lcc,
                                                             cfg.split ? nullptr : global);
    if (global && (!outputs || cfg.split)) global_kernel<<<1, 1, 0, s>>>(w.ctr, global);
    if (BATCH && graph_T) graph_triangles_kernel<<<gb, kThreads, 0, s>>>(w.gsum, w.graphs, graph_T);
    if (timing) cudaEventRecord(timing->ev[4], s);
    return cudaGetLastError() == cudaSuccess ? GTC_OK : GTC_ERR_CUDA;
}

}  // namespace

template <typename OffT>
gtc_status run_count(const OffT *off, const int *ind, long long n, long long nnz,
                     bool per_vertex, long long *r, long long *t, double *lcc,
                     long long *global, void *ws, size_t ws_bytes,
                     cudaStream_t stream, const RowConfig &cfg, CountTimings *timing,
                     const Batch *batch, const int *gate, Data *data)
{
    const long long graphs = batch ? batch->num_graphs : 0;
    const Plan p = make_plan(n, nnz, (int)sizeof(OffT) * 8, per_vertex, graphs);
    if (ws_bytes < p.need) return GTC_ERR_WORKSPACE_TOO_SMALL;
    char *base = static_cast<char *>(ws);
    NvtxRange count_range("gtc_count");
    // status word, counters, histograms and credits lead the workspace
    if (cudaMemsetAsync(base, 0, p.zero_bytes, stream) != cudaSuccess) return GTC_ERR_CUDA;
    View<OffT> w;
    w.off = off;
    w.ind = ind;
    w.n = n;
    w.nnz = nnz;
    w.vstart = batch ? batch->vstart : nullptr;
    w.graphs = graphs;
    w.word = (int)sizeof(unsigned int);
    w.gate = gate;
    w.bitmaps = cfg.dense && (batch || n <= kBitSpan);
    w.sparse = cfg.sparse && !batch;
    w.status = reinterpret_cast<unsigned int *>(base + p.o_status);
    w.ctr = reinterpret_cast<Counters *>(base + p.o_counters);
    w.recs = reinterpret_cast<GraphRec *>(base + p.o_recs);
    w.hist = reinterpret_cast<unsigned int *>(base + p.o_hist);
    w.key = reinterpret_cast<int *>(base + p.o_key);
    w.gid = reinterpret_cast<int *>(base + p.o_gid);
    w.vinfo = reinterpret_cast<VInfo *>(base + p.o_vinfo);
    w.find = reinterpret_cast<int *>(base + p.o_find);
    w.wide = reinterpret_cast<int *>(base + p.o_wide);
    w.litem = reinterpret_cast<int2 *>(base + p.o_litem);
    w.u = reinterpret_cast<unsigned int *>(base + p.o_u);
    w.ucap = (long long)(((ws_bytes < p.bytes ? ws_bytes : p.bytes) - p.o_u) / 4);
    w.tacc = per_vertex ? reinterpret_cast<unsigned long long *>(base + p.o_tacc) : nullptr;
    w.tcore = reinterpret_cast<unsigned long long *>(base + p.o_tcore);
    w.gsum = batch && batch->graph_T ? reinterpret_cast<unsigned long long *>(base + p.o_gsum)
                                     : nullptr;
    if (data) *data = w;
    if (n == 0) {
        if (timing)
            for (int i = 0; i < 5; ++i) cudaEventRecord(timing->ev[i], stream);
        if (global) global_kernel<<<1, 1, 0, stream>>>(w.ctr, global);
        if (batch && batch->graph_T &&
            cudaMemsetAsync(batch->graph_T, 0, sizeof(long long) * (size_t)graphs, stream) !=
                cudaSuccess)
            return GTC_ERR_CUDA;
        return cudaGetLastError() == cudaSuccess ? GTC_OK : GTC_ERR_CUDA;
    }
    const bool p32 = nnz < (1ll << 32);          // list positions fit 32 bits
    if (batch) {
        auto go = p32 ? launch<OffT, true, true, unsigned int> : launch<OffT, true, true, long long>;
        return go(w, GraphRec{}, r, t, lcc, global, batch->graph_T, stream, cfg, timing);
    }
    // the largest core whose bit matrix fits: u_row(k) <= ucap
    GraphRec lim;
    long long room = 0;
    for (long long step = kCoreMax; step > 0; step >>= 1)
        if (room + step <= kCoreMax && u_row((int)(room + step)) <= w.ucap) room += step;
    core_limits(n, nnz, room, lim.dmin, lim.long_min, lim.kcap);
    lim.nv = (int)n;
    auto go = per_vertex ? (p32 ? launch<OffT, false, true, unsigned int>
                                : launch<OffT, false, true, long long>)
                         : (p32 ? launch<OffT, false, false, unsigned int>
                                : launch<OffT, false, false, long long>);
    return go(w, lim, r, t, lcc, global, nullptr, stream, cfg, timing);
}

template gtc_status run_count<int>(const int *, const int *, long long, long long, bool,
                                   long long *, long long *, double *, long long *, void *,
                                   size_t, cudaStream_t, const RowConfig &, CountTimings *,
                                   const Batch *, const int *, Data *);
template gtc_status run_count<long long>(const long long *, const int *, long long, long long,
                                         bool, long long *, long long *, double *, long long *,
                                         void *, size_t, cudaStream_t, const RowConfig &,
                                         CountTimings *, const Batch *, const int *, Data *);

}  // namespace gtc
