// Row-major ("one writer per output row") schedule of the partitioned SpMM.
//
// At upload every partition's remote CSC block is transposed and merged with
// its local CSR, giving for each output row its entries in column order.
// Warps stream work items -- runs of rows, or segments of rows longer than a
// threshold ("hubs") -- gather the rows of X the entries name (16-byte
// vectors, UNROLL loads in flight per lane group), accumulate in FP32
// registers and write each output row once with plain stores: no atomics, no
// zeroing pass, the same summation order on every run, and BF16 output is
// rounded straight from the registers.  Hub segments go to an FP32 workspace;
// a second kernel adds each hub's partials pairwise (a binary tree in fixed
// order) and writes the row.
#pragma once
#include "spmm_kernels.cuh"

namespace cola {
namespace dev {

// Store E accumulated values to Y (FP32 or BF16), optionally adding the old
// contents (single writer, so a plain read-modify-write).
template <typename TY, int E, bool VEC_Y>
__device__ __forceinline__ void store_out(TY *p, const float (&a)[E], bool accumulate);

template <>
__device__ __forceinline__ void store_out<float, 4, true>(float *p, const float (&a)[4], bool accumulate)
{
    float4 v = make_float4(a[0], a[1], a[2], a[3]);
    if (accumulate) {
        const float4 o = *reinterpret_cast<const float4 *>(p);
        v.x += o.x;
        v.y += o.y;
        v.z += o.z;
        v.w += o.w;
    }
    __stcs(reinterpret_cast<float4 *>(p), v);  // Y is written once: evict-first in L2, X rows stay
}

template <>
__device__ __forceinline__ void store_out<float, 8, true>(float *p, const float (&a)[8], bool accumulate)
{
    const float lo[4] = {a[0], a[1], a[2], a[3]};
    const float hi[4] = {a[4], a[5], a[6], a[7]};
    store_out<float, 4, true>(p, lo, accumulate);
    store_out<float, 4, true>(p + 4, hi, accumulate);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b)
{
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);  // RNE; .x = a (low half)
    return *reinterpret_cast<uint32_t *>(&h);
}

template <>
__device__ __forceinline__ void store_out<__nv_bfloat16, 8, true>(__nv_bfloat16 *p, const float (&a)[8], bool)
{
    __stcs(reinterpret_cast<uint4 *>(p),
           make_uint4(pack_bf16x2(a[0], a[1]), pack_bf16x2(a[2], a[3]), pack_bf16x2(a[4], a[5]), pack_bf16x2(a[6], a[7])));
}

template <>
__device__ __forceinline__ void store_out<__nv_bfloat16, 4, true>(__nv_bfloat16 *p, const float (&a)[4], bool)
{
    *reinterpret_cast<uint2 *>(p) = make_uint2(pack_bf16x2(a[0], a[1]), pack_bf16x2(a[2], a[3]));
}

template <>
__device__ __forceinline__ void store_out<float, 2, true>(float *p, const float (&a)[2], bool accumulate)
{
    float2 v = make_float2(a[0], a[1]);
    if (accumulate) {
        const float2 o = *reinterpret_cast<const float2 *>(p);
        v.x += o.x;
        v.y += o.y;
    }
    __stcs(reinterpret_cast<float2 *>(p), v);
}

template <>
__device__ __forceinline__ void store_out<__nv_bfloat16, 2, true>(__nv_bfloat16 *p, const float (&a)[2], bool)
{
    *reinterpret_cast<uint32_t *>(p) = pack_bf16x2(a[0], a[1]);
}

template <>
__device__ __forceinline__ void store_out<float, 1, false>(float *p, const float (&a)[1], bool accumulate)
{
    *p = accumulate ? *p + a[0] : a[0];
}

template <>
__device__ __forceinline__ void store_out<__nv_bfloat16, 1, false>(__nv_bfloat16 *p, const float (&a)[1], bool)
{
    *p = __float2bfloat16_rn(a[0]);
}

// A lane's values one element at a time, STEP apart, as far as `left`: an output
// whose rows are not vector-aligned or end inside a vector.
template <typename TY, int E, int STEP = 1>
__device__ __forceinline__ void store_some(TY *p, const float (&a)[E], bool accumulate, int left)
{
#pragma unroll
    for (int q = 0; q < E; q++)
        if (q * STEP < left) {
            const float v[1] = {a[q]};
            store_out<TY, 1, false>(p + q * STEP, v, accumulate);
        }
}

// Work items of the streaming form, segments first, then tasks, one 16-byte
// descriptor each (a dependent chain of row pointers per item otherwise):
//   segment it:  entries [beg, beg + n) of one hub row; partial -> ws row it
//   task:        entries [beg, beg + n) of consecutive rows; out = position in
//                nz_row of the first of its rows that has entries
// An entry's column carries kRowEnd when it is the last of its row, so the
// stream needs no row pointers.  Rows without entries are in no item: every
// item writes its even share of their zeros at its end, beside other warps'
// gathers (0.04 of 1.07 ms on a scale-20 R-MAT graph at K = 128).
struct __align__(16) WorkItem {
    int64_t beg;
    int32_t n;
    int32_t out;
};

struct BlockArgs {
    const WorkItem *item;
    const int32_t *col;
    const float *val;
    const int32_t *nz_row;     // rows with entries, ascending
    const int32_t *empty_row;  // rows without, ascending
    int32_t nseg, nitem;  // items [0, nseg) segments, [nseg, nitem) tasks
    int32_t nempty, empty_share;  // rows without entries, and how many of them an item writes
    float *ws;            // nseg x K FP32 partials
    int64_t ld_ws;
    // Work-item counters for the dynamic schedule (kMaxItemQueues per-tile
    // counters, then the count of warps that have finished); all zero between
    // launches: the last warp of a launch resets them.  NULL: static
    // grid-stride assignment.
    unsigned int *queue;
};

// acc[q] += v * x[2q .. 2q+1] for one vector of X, with the packed FP32x2
// fused multiply-add of sm_100 (two products per instruction).
template <typename TR>
__device__ __forceinline__ void fma_vec2(float2 (&acc)[TR::E / 2], float2 vv, const typename TR::raw_t &r)
{
    float f[TR::E];
    TR::unpack(r, f);
#pragma unroll
    for (int q = 0; q < TR::E / 2; q++)
        acc[q] = __ffma2_rn(vv, make_float2(f[2 * q], f[2 * q + 1]), acc[q]);
}

__device__ __forceinline__ WorkItem load_item(const WorkItem *p)
{
    const int4 v = __ldg(reinterpret_cast<const int4 *>(p));
    WorkItem w;
    w.beg = (int64_t)(((uint64_t)(uint32_t)v.y << 32) | (uint32_t)v.x);
    w.n = v.z;
    w.out = v.w;
    return w;
}

// The current 32 entries of a warp: columns and values apart, so that 4 columns
// of a round are one 16-byte shared-memory load; each value twice, so that it
// is read as the register pair the packed FMA takes; and the output rows that
// end in the batch, in order.
struct __align__(16) EntryBatch {
    float2 val[32];
    int32_t col[32];
    int32_t row[32];
};

// base + c * stride bytes, one multiply-add.
__device__ __forceinline__ const char *row_at(const char *base, int32_t c, int32_t stride)
{
    unsigned long long r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(c), "r"(stride), "l"(base));
    return reinterpret_cast<const char *>(r);
}

// Lane id and warp in the block as values the compiler keeps (it re-reads
// threadIdx, a slow special register, inside the loops otherwise).
__device__ __forceinline__ int lane_id()
{
    int l;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(l));
    return l;
}
__device__ __forceinline__ unsigned int warp_in_block()
{
    unsigned int t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t >> 5;
}

// How an item's entries are summed: LG lanes cover one row tile of X (NV
// vectors each); G = 32 / LG lane groups take interleaved entries of the stream
// (group g takes entries g, g + G, ... of each 32-entry batch), so narrow rows
// still keep 32 lanes busy.  A round is G * UNROLL consecutive entries whose
// loads are all in flight; it is added up and cut where rows end.  At a row end
// the groups' sums are added in a butterfly that halves the features each lane
// holds at every step (about E shuffles a row instead of E log2 G), and each
// lane writes the features it is left with.
// What bounds it: the L1/L2 gather traffic of X with UNROLL x resident warps
// rows in flight; instruction issue comes next, so a round inside one row costs
// 3 shared loads, one address and one load per entry, and the products.
// Measured against the form that walked row pointers (R-MAT, one lane group a
// row, one product under ncu): scale 20, K = 128 FP32 1.084 -> 1.042 ms, scale 21,
// K = 256 BF16 3.94 -> 3.86; uniform rows of 20 entries at K = 100 83 -> 74 us;
// narrow rows: K = 16 BF16 206 -> 117 us, K = 32 FP32 on 16 K rows 23 -> 13 us.
// Slower (scale 20, K = 128 FP32, 1.07 ms in the same runs): 8 rows in
// flight at 3 blocks (1.10 ms), 2 at 5 or 6 (1.35), the next row's load issued
// as each row is added (1.64).
// VEC_Y: rows of Y are written in vectors; else (their start is not aligned or K
// ends inside a vector of X) element by element, X read in vectors or, with
// LooseTraits, element by element too.  RED: sums are added to Y with reductions
// (other warps add to the same rows).
template <typename TR, typename TY, int LG, int NV, int UNROLL, bool VEC_Y = true, bool RED = false>
struct RowStream {
    using T = typename ElemOf<TR>::T;
    using raw_t = typename TR::raw_t;
    static constexpr int E = TR::E;
    static constexpr int G = 32 / LG;
    static constexpr int R = G * UNROLL;  // entries per round
    static constexpr int LANES = LG, NVEC = NV;
    static constexpr bool LOOSE = kLoose<TR>;
    static constexpr int STEP = LOOSE ? LG : 1;  // between a lane's features of one vector
    static_assert(!LOOSE || (!VEC_Y && !RED), "element-wise X goes with element-wise Y");
    static_assert(32 % R == 0 && (NV == 1 || LG == 32), "rounds must divide the 32-entry batch");

    float2 acc[NV][E / 2];
    const char *xk;  // X + the lane's first feature
    int32_t ldxb;    // bytes between rows (the vector path's fit 31 bits)
    int64_t ldxe;    // elements between rows (LOOSE)
    TY *Y;
    int64_t ldy;
    int koff;  // the lane's first feature
    int K;
    int lane, g, gl;
    bool kok[NV];
    bool accumulate;
    bool to_ws;  // the current item's row goes to the workspace

    __device__ __forceinline__ void init(const T *X, int64_t ldx_, TY *Y_, int64_t ldy_, int K_, int k0, int acc_)
    {
        K = K_;
        lane = lane_id();
        g = lane / LG;
        gl = lane % LG;
        ldxb = (int32_t)(ldx_ * (int64_t)sizeof(T));
        ldxe = ldx_;
        ldy = ldy_;
        koff = k0 + gl * (LOOSE ? 1 : E);
        xk = reinterpret_cast<const char *>(X + koff);
        Y = Y_;
        accumulate = acc_ != 0;
#pragma unroll
        for (int j = 0; j < NV; j++)
            kok[j] = koff + j * LG * E < K;
    }

    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int j = 0; j < NV; j++)
#pragma unroll
            for (int q = 0; q < E / 2; q++)
                acc[j][q] = make_float2(0.f, 0.f);
    }

    // N values of a row of Y or, always in vectors, of the workspace.
    template <typename TO, int N>
    __device__ __forceinline__ void put(TO *p, const float (&a)[N], bool add, int left) const
    {
        if constexpr (RED)
            red_add<N, true>(p, a);
        else if constexpr (LOOSE)
            store_some<TO, N, STEP>(p, a, add, left);
        else if constexpr (VEC_Y)
            store_out<TO, N, (N > 1)>(p, a, add);
        else if (to_ws)
            store_out<TO, N, (N > 1)>(p, a, false);
        else
            store_some<TO, N>(p, a, add, left);
    }

    // The warp's sums to one row of Y or of the workspace (p: the lane's first
    // feature in that row); clears them.
    template <typename TO>
    __device__ __forceinline__ void write_row(TO *p, bool add)
    {
        if constexpr (G == 1) {
#pragma unroll
            for (int j = 0; j < NV; j++) {
                float a[E];
#pragma unroll
                for (int q = 0; q < E / 2; q++) {
                    a[2 * q] = acc[j][q].x;
                    a[2 * q + 1] = acc[j][q].y;
                }
                if (kok[j])
                    put(p + j * LG * E, a, add, K - koff - j * LG * E);
            }
        } else {
            float v[E];
#pragma unroll
            for (int q = 0; q < E / 2; q++) {
                v[2 * q] = acc[0][q].x;
                v[2 * q + 1] = acc[0][q].y;
            }
            // step `off`: the lane keeps the half its bit selects and adds the
            // partner's, the same pairs in the same order as a full exchange
            int f = 0;
#pragma unroll
            for (int off = LG, cnt = E; off < 32; off <<= 1, cnt = cnt > 1 ? cnt / 2 : 1) {
                if (cnt > 1) {
                    const bool up = (lane & off) != 0;
#pragma unroll
                    for (int q = 0; q < E / 2; q++)
                        if (q < cnt / 2) {
                            const float send = up ? v[q] : v[q + cnt / 2];
                            const float keep = up ? v[q + cnt / 2] : v[q];
                            v[q] = keep + __shfl_xor_sync(kFull, send, off);
                        }
                    f += up ? cnt / 2 : 0;
                } else {
                    v[0] += __shfl_xor_sync(kFull, v[0], off);
                }
            }
            constexpr int EO = E / G > 0 ? E / G : 1;     // features a lane is left with
            constexpr int kDup = E >= G ? 0 : 32 - LG * E;  // lane bits of the steps past one feature: copies
            if (kok[0] && (lane & kDup) == 0) {
                float a[EO];
#pragma unroll
                for (int q = 0; q < EO; q++)
                    a[q] = v[q];
                put(p + f * STEP, a, add, K - koff - f * STEP);
            }
        }
        clear();
    }

    template <bool ALL>
    __device__ __forceinline__ void load_round(const EntryBatch &eb, int jj, int cnt, raw_t (&xr)[UNROLL][NV]) const
    {
        int32_t c[UNROLL];
        if constexpr (G == 1 && UNROLL % 4 == 0) {
#pragma unroll
            for (int u = 0; u < UNROLL; u += 4) {
                const int4 v = *reinterpret_cast<const int4 *>(eb.col + jj + u);
                c[u] = v.x;
                c[u + 1] = v.y;
                c[u + 2] = v.z;
                c[u + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int u = 0; u < UNROLL; u++)
                c[u] = eb.col[jj + u * G + g];
        }
#pragma unroll
        for (int u = 0; u < UNROLL; u++) {
            if (ALL || u * G + g < cnt) {
                if constexpr (LOOSE) {
                    const T *xp = reinterpret_cast<const T *>(xk) + (int64_t)c[u] * ldxe;
#pragma unroll
                    for (int j = 0; j < NV; j++)
                        xr[u][j] = TR::load(xp + j * LG * E, LG, K - koff - j * LG * E);
                } else {
                    const T *xp = reinterpret_cast<const T *>(row_at(xk, c[u], ldxb));
#pragma unroll
                    for (int j = 0; j < NV; j++)
                        if (kok[j])
                            xr[u][j] = TR::load(xp + j * LG * E);
                }
            }
        }
    }

    __device__ __forceinline__ void round_values(const EntryBatch &eb, int jj, float2 (&v)[UNROLL]) const
    {
        if constexpr (G == 1 && UNROLL % 2 == 0) {
#pragma unroll
            for (int u = 0; u < UNROLL; u += 2) {
                const float4 w = *reinterpret_cast<const float4 *>(eb.val + jj + u);
                v[u] = make_float2(w.x, w.y);
                v[u + 1] = make_float2(w.z, w.w);
            }
        } else {
#pragma unroll
            for (int u = 0; u < UNROLL; u++)
                v[u] = eb.val[jj + u * G + g];
        }
    }

    // One batch of n entries (1..32); ends: bit i set where entry i is its
    // row's last; rows: the rows that end, in order.
    __device__ __forceinline__ void batch(const EntryBatch &eb, const int32_t *rows, const int n, const uint32_t ends)
    {
        auto flush = [&]() {
            const int row = *rows++;
            write_row(Y + (int64_t)row * ldy + koff, accumulate);
        };
#pragma unroll 1
        for (int jj = 0; jj < n; jj += R) {
            raw_t xr[UNROLL][NV];
            const int cnt = min(R, n - jj);
            uint32_t e = ends >> jj;
            if (R < 32)
                e &= (1u << (R & 31)) - 1u;
            if (cnt == R)
                load_round<true>(eb, jj, R, xr);
            else
                load_round<false>(eb, jj, cnt, xr);
            float2 v[UNROLL];
            round_values(eb, jj, v);
            if (cnt == R && e == 0) {
#pragma unroll
                for (int u = 0; u < UNROLL; u++)
#pragma unroll
                    for (int j = 0; j < NV; j++)
                        fma_vec2<TR>(acc[j], v[u], xr[u][j]);
            } else if constexpr (G == 1 && UNROLL <= 4) {
                // entry by entry: a row ends after the entries marked in e
#pragma unroll
                for (int u = 0; u < UNROLL; u++) {
                    if (u < cnt) {
#pragma unroll
                        for (int j = 0; j < NV; j++)
                            fma_vec2<TR>(acc[j], v[u], xr[u][j]);
                    }
                    if (e & (1u << u))
                        flush();
                }
            } else if constexpr (G == 2 && E <= 4 && UNROLL <= 4) {
                // pair by pair: a row ends after the first or the second of a pair
#pragma unroll
                for (int u = 0; u < UNROLL; u++) {
                    const uint32_t p = (e >> (2 * u)) & 3u;
                    const bool have = 2 * u + g < cnt;
                    auto add = [&]() {
#pragma unroll
                        for (int j = 0; j < NV; j++)
                            fma_vec2<TR>(acc[j], v[u], xr[u][j]);
                    };
                    if (have && (g == 0 || !(p & 1u)))
                        add();
                    if (p & 1u) {
                        flush();
                        if (have && g == 1)
                            add();
                    }
                    if (p & 2u)
                        flush();
                }
            } else if constexpr (G > 1 && UNROLL > 1) {
                // one entry per group at a time, cut where rows end among them
#pragma unroll
                for (int u = 0; u < UNROLL; u++) {
                    uint32_t p = (e >> (u * G)) & ((1u << G) - 1u);
                    const bool have = u * G + g < cnt;
                    int lo = 0;
                    while (p) {
                        const int sh = __ffs(p);
                        if (have && g >= lo && g < sh) {
#pragma unroll
                            for (int j = 0; j < NV; j++)
                                fma_vec2<TR>(acc[j], v[u], xr[u][j]);
                        }
                        flush();
                        p &= p - 1;
                        lo = sh;
                    }
                    if (have && g >= lo) {
#pragma unroll
                        for (int j = 0; j < NV; j++)
                            fma_vec2<TR>(acc[j], v[u], xr[u][j]);
                    }
                }
            } else {
                // cut the round at the row ends it contains
                int lo = 0;
                while (true) {
                    const int sh = e ? __ffs(e) : cnt;
#pragma unroll
                    for (int u = 0; u < UNROLL; u++) {
                        const int i = u * G + g;
                        if (i >= lo && i < sh) {
#pragma unroll
                            for (int j = 0; j < NV; j++)
                                fma_vec2<TR>(acc[j], v[u], xr[u][j]);
                        }
                    }
                    if (!e)
                        break;
                    flush();
                    e &= e - 1;
                    lo = sh;
                    if (lo >= cnt)
                        break;
                }
            }
        }
    }
};

// One work item.  While a batch is summed the next one's entries are on their
// way in registers.  before_x() runs when the first entries are under way and
// before X is read or anything written.
template <typename RS, typename F>
__device__ __forceinline__ void stream_item(RS &rs, const BlockArgs &ba, const int it, EntryBatch &eb, F before_x)
{
    const int lane = rs.lane;
    const bool seg = it < ba.nseg;
    rs.to_ws = seg;
    const WorkItem w = load_item(ba.item + it);
    int64_t pos = w.beg + lane;
    int left = w.n;
    int kpos = w.out + lane;
    int mc = 0, mr = 0;
    float mv = 0.f;
    auto fetch = [&]() {
        // the entry stream is read once: evict-first, so it does not push X rows out of L2
        if (lane < left) {
            mc = __ldcs(ba.col + pos);
            mv = __ldcs(ba.val + pos);
        }
        if (!seg)
            mr = __ldg(ba.nz_row + kpos);  // the list is padded by 32
    };
    fetch();
    before_x();
    rs.clear();
    while (left > 0) {
        const int n = min(32, left);
        const uint32_t ends = seg ? 0u : __ballot_sync(kFull, mc < 0 && lane < n);
        __syncwarp();
        eb.col[lane] = mc & kColMask;
        eb.val[lane] = make_float2(mv, mv);
        eb.row[lane] = mr;
        __syncwarp();
        left -= 32;
        pos += 32;
        kpos += __popc(ends);
        if (left > 0)
            fetch();
        rs.batch(eb, eb.row, n, ends);
    }
    if (seg)
        rs.write_row(ba.ws + (int64_t)it * ba.ld_ws + rs.koff, false);
    // this item's share of the empty rows, G rows at a time
    if (ba.nempty > 0 && !rs.accumulate) {
        rs.to_ws = false;
        const int64_t z0 = (int64_t)it * ba.empty_share;
        const int zn = (int)min((int64_t)ba.empty_share, ba.nempty - z0);
        for (int i = rs.g; i < zn; i += RS::G) {
            const int row = __ldg(ba.empty_row + z0 + i);
            const float z[RS::E] = {};
#pragma unroll
            for (int j = 0; j < RS::NVEC; j++)
                if (rs.kok[j])
                    rs.put(rs.Y + (int64_t)row * rs.ldy + rs.koff + j * RS::LANES * RS::E, z, false,
                           rs.K - rs.koff - j * RS::LANES * RS::E);
        }
        __syncwarp();
    }
}

// The item after the one being drawn: the first one of every warp is its own
// number, the others come from the counter.
__device__ __forceinline__ unsigned int draw_item(unsigned int *queue, unsigned int nwarps)
{
    return nwarps + atomicAdd(queue, 1u);
}

// All items of one feature tile, drawn by this warp, one ahead, so that the
// atomic's latency hides behind the current item.  The grid may have started
// before the kernel in front of it has ended: only the graph's own arrays, which
// no kernel writes, are read before pdl_wait.
template <typename RS, bool DYN>
__device__ __forceinline__ void stream_items(RS &rs, const BlockArgs &ba, const unsigned int warp,
                                             const unsigned int nwarps, EntryBatch &eb,
                                             unsigned int *queue)
{
    const unsigned int total = (unsigned int)ba.nitem;
    // with at most one item per warp nothing is drawn (item_queue_release agrees)
    const bool draw = DYN && total > nwarps;
    for (unsigned int it = warp; it < total;) {
        unsigned int next = DYN ? total : it + nwarps;
        stream_item(rs, ba, (int)it, eb, [&]() {
            if (it == warp)
                pdl_wait();
            if (draw && rs.lane == 0)
                next = draw_item(queue, nwarps);
        });
        it = draw ? __shfl_sync(kFull, next, 0) : next;
    }
}

// End of a launch with the dynamic schedule: the last of `warps` warps to
// finish puts the item counters back to zero for the next launch (every warp
// has drawn its final item before it counts itself finished).
__device__ __forceinline__ void item_queue_release(unsigned int *queue, const unsigned int nqueues,
                                                   unsigned int *finished, const unsigned int warps)
{
    if ((threadIdx.x & 31) == 0) {
        if (atomicAdd(finished, 1u) == warps - 1) {
            for (unsigned t = 0; t < nqueues; t++)
                atomicExch(queue + t, 0u);
            atomicExch(finished, 0u);
        }
    }
}

template <typename TR, typename TY, int LG, int NV, int UNROLL, int MINB = 1, bool DYN = false, bool VEC_Y = true>
__global__ void __launch_bounds__(kThreads, MINB) rowblock_spmm_kernel(const __grid_constant__ BlockArgs ba,
                                                                       const typename ElemOf<TR>::T *__restrict__ X,
                                                                       int64_t ldx, TY *__restrict__ Y, int64_t ldy,
                                                                       int K, int accumulate)
{
    __shared__ EntryBatch s_ent[kWarpsPerBlock];
    pdl_launch_dependents();
    constexpr int W = LG * NV * TR::E;
    const int k0 = blockIdx.y * W;
    const unsigned int nwarps = gridDim.x * kWarpsPerBlock, wb = warp_in_block();
    RowStream<TR, TY, LG, NV, UNROLL, VEC_Y> rs;
    rs.init(X, ldx, Y, ldy, K, k0, accumulate);
    stream_items<RowStream<TR, TY, LG, NV, UNROLL, VEC_Y>, DYN>(rs, ba, blockIdx.x * kWarpsPerBlock + wb, nwarps, s_ent[wb],
                                                         DYN ? ba.queue + blockIdx.y : nullptr);
    if (DYN && (unsigned int)ba.nitem > nwarps)
        item_queue_release(ba.queue, gridDim.y, ba.queue + kMaxItemQueues, nwarps * gridDim.y);
}

// The same schedule with the feature tiles one after another instead of side
// by side (blockIdx.y): the grid sweeps every item of tile 0, then of tile 1,
// ..., so the X columns being gathered at any moment are one tile wide.  Every
// element's sum is the same chain of FMAs whichever tile width computes it
// (one lane group per row: LG = 32).
template <typename TR, typename TY, int NV, int UNROLL, int MINB = 1>
__global__ void __launch_bounds__(kThreads, MINB) rowblock_tiled_kernel(const __grid_constant__ BlockArgs ba,
                                                                        const typename ElemOf<TR>::T *__restrict__ X,
                                                                        int64_t ldx, TY *__restrict__ Y, int64_t ldy,
                                                                        int K, int accumulate)
{
    __shared__ EntryBatch s_ent[kWarpsPerBlock];
    pdl_launch_dependents();
    constexpr int W = 32 * NV * TR::E;
    const unsigned int nwarps = gridDim.x * kWarpsPerBlock;
    // tile t starts where the last one's round robin over the warps ended
    unsigned int warp = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    for (int k0 = 0; k0 < K; k0 += W) {
        RowStream<TR, TY, 32, NV, UNROLL> rs;
        rs.init(X, ldx, Y, ldy, K, k0, accumulate);
        stream_items<RowStream<TR, TY, 32, NV, UNROLL>, false>(rs, ba, warp, nwarps, s_ent[threadIdx.x >> 5],
                                                               nullptr);
        warp = (warp + nwarps - (unsigned int)ba.nitem % nwarps) % nwarps;
    }
}

// Hub rows (workspace rows are 16-byte aligned and whole vectors): a group of lc
// lanes (32, or the power of two that covers K / 4 below) owns one (hub, 4 *
// lc-feature tile).  The m partials are added pairwise in the order of a binary
// counter: partial i closes the running block sums of sizes 1, 2, 4,
// ... that its index's trailing one bits name, and the open blocks at the end
// are folded larger (earlier) first.  The counter is run kHubRadix partials at a
// time, all their loads in flight and every running sum in a register: whole
// blocks of kHubRadix are reduced to one value each in the workspace, blocks of
// those to kHubRadix^2, and so on; then the open blocks of every power are
// folded.  Hubs of kHubTeam or more partials are left to the end and each shared
// by the whole block: one lane group alone walks 240 partials in 55 us, which
// was the tail of the launch.  Measured in the step, launch included: 16 K rows
// at K = 32 6.7 -> 2.6 us, 524 K rows at K = 16 27 -> 10, scale 20 at K = 128
// 56 -> 33.  Teams from 32 partials on: below, one group's few rounds cost less
// than the block's waits.
constexpr int kHubRadixBits = 3, kHubRadix = 1 << kHubRadixBits;
constexpr int kHubTeam = 32;
constexpr int kHubList = 128;  // long hubs a block keeps for its end; more are walked alone

// Counter over p[0 .. cnt) (stride ld floats, cnt <= kHubRadix).  FULL: tot =
// the block's sum.  Otherwise folds the open blocks into tot (any: tot already
// holds a sum).
template <bool FULL>
__device__ __forceinline__ void hub_counter(const float *p, const int64_t ld, const int cnt, float4 &tot, bool &any)
{
    float4 v[kHubRadix];
#pragma unroll
    for (int i = 0; i < kHubRadix; i++, p += ld)
        if (FULL || i < cnt)
            v[i] = __ldcg(reinterpret_cast<const float4 *>(p));
    auto add = [](float4 a, float4 c) {
        return make_float4(a.x + c.x, a.y + c.y, a.z + c.z, a.w + c.w);
    };
    // v[i] becomes the block that partial i closes; v[j] stays the open block ending at j
    static_assert(kHubRadix == 8, "the blocks are spelled out");
#define COLA_CLOSE(i, l)        \
    if (FULL || (i) < cnt)      \
        v[i] = add(v[(i) - (l)], v[i])
    COLA_CLOSE(1, 1);
    COLA_CLOSE(3, 1);
    COLA_CLOSE(5, 1);
    COLA_CLOSE(7, 1);
    COLA_CLOSE(3, 2);
    COLA_CLOSE(7, 2);
    COLA_CLOSE(7, 4);
#undef COLA_CLOSE
    if (FULL) {
        tot = v[kHubRadix - 1];
        return;
    }
    auto pick = [](bool c, float4 a, float4 b) {
        return make_float4(c ? a.x : b.x, c ? a.y : b.y, c ? a.z : b.z, c ? a.w : b.w);
    };
    auto fold = [&](float4 b) {
        tot = any ? add(tot, b) : b;
        any = true;
    };
    const bool c4 = cnt & 4, c2 = cnt & 2;
    if (c4)
        fold(v[3]);
    if (c2)
        fold(pick(c4, v[5], v[1]));
    if (cnt & 1)
        fold(pick(c4, pick(c2, v[6], v[4]), pick(c2, v[2], v[0])));
}

// One hub's tile of one output.
template <typename TY>
struct HubItem {
    const int32_t *hub_row;
    const int64_t *hub_seg;
    int64_t h;
    int tile;
    float *ws;
    int64_t ld_ws;
    TY *Y;
    int64_t ldy;
    int K;
    __device__ __forceinline__ int partials() const { return (int)(__ldg(hub_seg + h + 1) - __ldg(hub_seg + h)); }
};

// One item by `teams` lane groups of which this is number `team`: the m partials
// at wp (rows of ld floats; this lane's 4 features) to y.  One copy of the code
// for both kinds of call.  A lane re-reads the sums of its own features only;
// with several teams the block waits between powers.
template <typename TY, bool VEC_Y>
__device__ __noinline__ void hub_combine_item(float *wp, const int64_t ld, const int m, TY *y, const int left,
                                              const int accumulate, const int team, const int teams)
{
    const bool kok = left > 0;
    float4 tot = make_float4(0.f, 0.f, 0.f, 0.f);
    bool any = false;
    // whole blocks of kHubRadix^1, ^2, ... partials: each block's sum over its first partial
    int power = 0;  // log2 of the partials per element
    for (int n = m >> kHubRadixBits; n > 0; n >>= kHubRadixBits, power += kHubRadixBits) {
        if (kok)
#pragma unroll 1
            for (int c = team; c < n; c += teams) {
                float *p = wp + ((int64_t)c << (power + kHubRadixBits)) * ld;
                float4 b;
                hub_counter<true>(p, ld << power, kHubRadix, b, any);
                __stcg(reinterpret_cast<float4 *>(p), b);
            }
        if (teams > 1)
            __syncthreads();
    }
    if (team != 0 || !kok)
        return;
    // the open blocks, larger powers (earlier partials) first
    int base = 0;
#pragma unroll 1
    for (; power >= 0; power -= kHubRadixBits) {
        const int cnt = (m - base) >> power;
        if (cnt > 0)
            hub_counter<false>(wp + base * ld, ld << power, cnt, tot, any);
        base += cnt << power;
    }
    const float r[4] = {tot.x, tot.y, tot.z, tot.w};
    if constexpr (VEC_Y)
        store_out<TY, 4, true>(y, r, accumulate != 0);
    else
        store_some<TY, 4>(y, r, accumulate != 0, left);
}

// Lanes per (hub, tile) of the combine and tiles per hub.
__host__ __device__ inline int hub_lanes(int K) { return K > 64 ? 32 : K > 32 ? 16 : K > 16 ? 8 : 4; }
__host__ __device__ inline int hub_tiles(int K) { return (K + 127) / 128; }

// Combine items [0, total) with `lc` lanes each; find(w) names item w.
// Neighbouring items (in R-MAT order: hubs of like length) go to different
// blocks.
template <typename TY, bool VEC_Y, typename FIND>
__device__ __forceinline__ void hub_combine_all(const int64_t total, const int lc, const int accumulate, FIND find)
{
    __shared__ int64_t s_big[kHubList];
    __shared__ int s_nbig;
    if (threadIdx.x == 0)
        s_nbig = 0;
    __syncthreads();
    const int groups = kThreads / lc, grp = threadIdx.x / lc, gl = threadIdx.x % lc;
    const unsigned int mask = lc == 32 ? kFull : ((1u << lc) - 1u) << ((threadIdx.x & 31) / lc * lc);
    auto combine = [&](const HubItem<TY> &it, int m, int team, int teams) {
        const int k = it.tile * 128 + gl * 4;
        hub_combine_item<TY, VEC_Y>(it.ws + __ldg(it.hub_seg + it.h) * it.ld_ws + k, it.ld_ws, m,
                             it.Y + (int64_t)__ldg(it.hub_row + it.h) * it.ldy + k, it.K - k, accumulate, team, teams);
    };
    for (int64_t w = (int64_t)grp * gridDim.x + blockIdx.x; w < total; w += (int64_t)gridDim.x * groups) {
        const HubItem<TY> it = find(w);
        const int m = it.partials();
        if (m >= kHubTeam) {
            int at = 0;
            if (gl == 0)
                at = atomicAdd(&s_nbig, 1);
            at = __shfl_sync(mask, at, 0, lc);
            if (at < kHubList) {
                if (gl == 0)
                    s_big[at] = w;
                continue;
            }
        }
        combine(it, m, 0, 1);
    }
    __syncthreads();
    const int nbig = min(s_nbig, kHubList);
    for (int q = 0; q < nbig; q++) {
        const HubItem<TY> it = find(s_big[q]);
        combine(it, it.partials(), grp, groups);
    }
}

template <typename TY, bool VEC_Y>
__global__ void __launch_bounds__(kThreads, 4) hub_combine_vec_kernel(const int32_t *__restrict__ hub_row,
                                                                  const int64_t *__restrict__ hub_seg, int64_t nhub,
                                                                  float *ws, int64_t ld_ws, TY *__restrict__ Y,
                                                                  int64_t ldy, int K, int accumulate)
{
    pdl_launch_dependents();
    pdl_wait();  // the partials
    const int tiles = hub_tiles(K);
    hub_combine_all<TY, VEC_Y>(nhub * tiles, hub_lanes(K), accumulate, [&](int64_t w) {
        return HubItem<TY>{hub_row, hub_seg, w / tiles, (int)(w % tiles), ws, ld_ws, Y, ldy, K};
    });
}

// X with every row padded to whole 16-byte vectors (zeros), for the vector form
// when K or the rows' alignment does not allow it: one thread per vector.
template <typename T>
__global__ void __launch_bounds__(kThreads) pad_rows_kernel(const T *__restrict__ X, int64_t ldx, T *__restrict__ P,
                                                           int nvec, int64_t total, int K)
{
    constexpr int E = 16 / sizeof(T);
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < total; i += (int64_t)gridDim.x * kThreads) {
        const int64_t r = i / nvec;
        const int k = (int)(i - r * nvec) * E;
        const T *p = X + r * ldx + k;
        __align__(16) T v[E];
#pragma unroll
        for (int q = 0; q < E; q++)
            v[q] = k + q < K ? __ldg(p + q) : T(0.f);
        *reinterpret_cast<uint4 *>(P + i * E) = *reinterpret_cast<const uint4 *>(v);
    }
}

}  // namespace dev
}  // namespace cola
