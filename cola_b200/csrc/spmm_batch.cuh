// Batched form: many graphs, each with its own X, Y and feature width.  Graphs
// are grouped by the lane width of their features (the geometry the
// single-graph kernel has for that width, so a graph's result is the same bits
// either way); each group is one persistent launch, and a group's blocks start
// as the blocks of the group before it end, so the launches have one tail
// between them.  Work items of a group's graphs are concatenated (graph g owns
// items [item0, item0 + nitem)); a warp finds its graph by advancing through the
// descriptor table (its items only increase).  With DYN the items are drawn from
// a counter (one ahead, as in the single-graph kernel): items differ in cost
// with the width, so a static share leaves warps idle.
#pragma once
#include "spmm_rows.cuh"

namespace cola {
namespace dev {

struct BatchGraph {
    BlockArgs ba;  // row view, items, workspace of this graph
    const void *X;
    int64_t ldx;
    void *Y;
    int64_t ldy;
    int32_t K;
    int32_t lg;    // lanes per row tile (row_lanes(K, E)), 64: 32 lanes, two vectors each
    int64_t item0; // first work item of this graph in its group's launch
    int64_t hub0;  // first combine item (hub x 128-feature tile) of this graph
    const int32_t *hub_row;
    const int64_t *hub_seg;
    int64_t nhub;
};

template <typename TR, typename TY, int LG, int NV, int UNROLL, int MINB, bool DYN>
__global__ void __launch_bounds__(kThreads, MINB) batch_rowblock_kernel(const BatchGraph *__restrict__ gs, int ng,
                                                                     unsigned int total, int accumulate,
                                                                     unsigned int *queue, unsigned int *finished)
{
    using T = typename ElemOf<TR>::T;
    __shared__ EntryBatch s_ent[kWarpsPerBlock];
    pdl_launch_dependents();
    const unsigned int wb = warp_in_block();
    EntryBatch &eb = s_ent[wb];
    const unsigned int nwarps = gridDim.x * kWarpsPerBlock;
    const int lane = lane_id();
    const bool draw = DYN && total > nwarps;
    int gi = 0;
    unsigned int it = blockIdx.x * kWarpsPerBlock + wb;
    while (it < total) {
        unsigned int next = 0;
        if (draw && lane == 0)
            next = draw_item(queue, nwarps);
        while (gi + 1 < ng && it >= gs[gi + 1].item0)
            gi++;
        const BatchGraph &bg = gs[gi];
        const int li = (int)(it - bg.item0);
        constexpr int W = LG * NV * TR::E;  // features per tile
        for (int k0 = 0; k0 < bg.K; k0 += W) {
            RowStream<TR, TY, LG, NV, UNROLL> rs;
            rs.init(static_cast<const T *>(bg.X), bg.ldx, static_cast<TY *>(bg.Y), bg.ldy, bg.K, k0, accumulate);
            stream_item(rs, bg.ba, li, eb, []() {});
        }
        it = draw ? __shfl_sync(kFull, next, 0) : it + nwarps;
    }
    if (draw)
        item_queue_release(queue, 1, finished, nwarps);
    pdl_wait();  // this grid ends after the group before it
}

template <typename TY>
__global__ void __launch_bounds__(kThreads, 4) batch_hub_combine_kernel(const BatchGraph *__restrict__ gs, int ng,
                                                                    int64_t total, int lanes, int accumulate)
{
    pdl_wait();  // the partials
    int gi = 0;
    hub_combine_all<TY, true>(total, lanes, accumulate, [&](int64_t w) {
        if (w < gs[gi].hub0)
            gi = 0;
        while (gi + 1 < ng && w >= gs[gi + 1].hub0)
            gi++;
        const BatchGraph &bg = gs[gi];
        const int tiles = hub_tiles(bg.K);
        const int64_t lw = w - bg.hub0;
        return HubItem<TY>{bg.hub_row, bg.hub_seg, lw / tiles, (int)(lw % tiles), bg.ba.ws, bg.ba.ld_ws,
                           static_cast<TY *>(bg.Y), bg.ldy, bg.K};
    });
}

}  // namespace dev
}  // namespace cola
