// gtc_core.cuh -- host interface of the counting pipeline.
#pragma once

#include "gtc_internal.cuh"

namespace gtc {

struct Data;

// Launch plan of one count.
struct RowConfig {
    // Large heavy graphs (mean degree > 24): wide and short rows in launches
    // of their own; otherwise one launch takes both.  gtc_tuning.labels.
    bool split = false;
    // Rows so long (mean degree >= 128, the graph not all core) that some are
    // looked up in bitmaps, by a kernel of their own.
    bool dense = false;
    // Mean degree of at most 4, a large graph: if it is uniform, its short rows'
    // pairs are looked up one by one, by a core kernel of its own.
    bool sparse = false;
};

// Kernel launches of one run_count with this configuration (the epilogue
// kernels counted as launched).
int launches_per_count(const RowConfig &cfg, bool per_vertex, long long n);

// Apply caller overrides (gtc_tuning, 0 = keep) to cfg; GTC_ERR_INVALID_ARGUMENT
// for a value outside the documented ranges.
gtc_status apply_tuning(RowConfig &cfg, const gtc_tuning *tuning);

// Optional CUDA events recorded between the pipeline phases:
// ev[0] start, ev[1] forward lists built, ev[2] table kernels done,
// ev[3] bit-matrix kernels done, ev[4] epilogue done.
struct CountTimings {
    cudaEvent_t ev[5];
};

// A batch: the vertex space is cut into graphs (vstart[0..G], device) whose
// neighbour ids are graph-local; graph_T (device, nullable) receives each
// graph's triangles.
struct Batch {
    const long long *vstart = nullptr;
    long long num_graphs = 0;
    long long *graph_T = nullptr;
};

// Workspace layout.  `need` is what a count must be given; `bytes` adds the
// bit matrix at its full size.  A count given less uses a smaller core.
struct Plan {
    size_t o_status = 0, o_counters = 0, o_recs = 0, o_hist = 0, o_tacc = 0, o_tcore = 0,
           o_gsum = 0, o_key = 0, o_gid = 0, o_vinfo = 0, o_find = 0, o_wide = 0, o_litem = 0,
           o_u = 0;
    size_t zero_bytes = 0;     // leading bytes that start at zero
    size_t need = 0, bytes = 0;
};

Plan make_plan(long long n, long long nnz, int off_bits, bool per_vertex, long long graphs = 0);

RowConfig pick_row_config(long long n, long long nnz);

// gate: device flag (nullable); while it is 0 the kernels end at once.  data
// (nullable) receives where the count's arrays are.
template <typename OffT>
gtc_status run_count(const OffT *off, const int *ind, long long n, long long nnz,
                     bool per_vertex, long long *r, long long *t, double *lcc,
                     long long *global, void *ws, size_t ws_bytes,
                     cudaStream_t stream, const RowConfig &cfg,
                     CountTimings *timing, const Batch *batch = nullptr,
                     const int *gate = nullptr, Data *data = nullptr);

}  // namespace gtc
