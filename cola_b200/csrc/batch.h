// Internal: the batched launch shared by the batched form and the server.
#pragma once
#include <algorithm>

#include "graph.h"
#include "spmm_batch.cuh"

namespace cola {

// Lane widths 1, 2, 4, 8, 16, 32, and 64 for two vectors a lane.
constexpr int kBatchGroups = 7;

// The graphs of one lane width: descriptors [first, first + count) of the
// table, `items` work items.
struct BatchGroup {
    int lg, first, count;
    int64_t items;
};

// One batched run over a device table of graph descriptors, sorted by lane
// width (build_groups).
struct BatchLaunch {
    const dev::BatchGraph *desc;
    int ngraphs;
    BatchGroup group[kBatchGroups];
    int ngroups;
    int64_t total_hub;
    int kmax;             // widest graph
    cola_dtype xdt, ydt;
    int unroll, grid_pct, accumulate;
    int blocks_per_sm;  // resident blocks per SM the streaming kernel is compiled for: 3 or 4
    // kBatchQueueBytes of counters at the end of the descriptor table's
    // allocation, zero between launches, or NULL for the static assignment;
    // launches that share counters must not overlap
    unsigned int *queue;
};

// Bytes of work-item counters a descriptor table's allocation carries after
// the descriptors (at a 256-byte aligned offset: batch_queue_offset).
constexpr size_t kBatchQueueBytes = 512;
inline size_t batch_queue_offset(size_t desc_bytes) { return (desc_bytes + 255) & ~(size_t)255; }

cola_status launch_batch(const BatchLaunch &L, cudaStream_t st);

// Sorts n descriptors by lane width (stable), numbers their work and combine
// items and fills in L's groups, total_hub and kmax.
cola_status build_groups(dev::BatchGraph *d, int n, BatchLaunch &L);

// Row view of graph g with hub workspace ws (rows of ld_ws floats) and the
// graph's own item counters.
inline dev::BlockArgs block_args(const cola_graph *g, float *ws, int64_t ld_ws)
{
    dev::BlockArgs ba;
    ba.item = static_cast<const dev::WorkItem *>(g->items);
    ba.col = g->rv_col;
    ba.val = g->rv_val;
    ba.nz_row = g->nz_row;
    ba.empty_row = g->empty_row;
    ba.nseg = (int32_t)g->nseg;
    ba.nitem = (int32_t)(g->nseg + g->ntask);
    ba.nempty = (int32_t)g->nempty;
    ba.empty_share = (int32_t)((g->nempty + std::max(ba.nitem, 1) - 1) / std::max(ba.nitem, 1));
    ba.ws = ws;
    ba.ld_ws = ld_ws;
    ba.queue = g->item_queue;
    return ba;
}

// What one row-major product of a graph needs beside its operands: hub partials
// (nseg rows of rows_ld_ws floats), room for the padded copy of X (rows_pad_bytes,
// or NULL: X is read as it is), and dev::kMaxItemQueues + 1 work-item counters,
// zero between products.  Products that share them must be ordered.
struct RowsWork {
    float *hub;
    void *x_pad;
    unsigned int *queue;
};
// Rows of the hub workspace are whole vectors of X.
inline int64_t rows_ld_ws(cola_dtype xdt, int K)
{
    const int64_t E = xdt == COLA_FLOAT32 ? 4 : 8;
    return (K + E - 1) / E * E;
}
size_t rows_pad_bytes(const cola_graph *g, cola_dtype xdt, const void *X, int64_t ldx, int K);
cola_status rows_product(const cola_graph *g, const RowsWork &w, const void *X, cola_dtype xdt, int64_t ldx, void *Y,
                         cola_dtype ydt, int64_t ldy, int K, const cola_spmm_opts *opts, cudaStream_t st);

// Descriptor of graph g with these operands and hub workspace (item0 / hub0
// left zero).
void fill_batch_graph(dev::BatchGraph &d, const cola_graph *g, const void *X, int64_t ldx, void *Y, int64_t ldy,
                      int32_t K, cola_dtype xdt, float *ws);

}  // namespace cola
