// The fused partitioned SpMM over the split chunks (spmm_kernels.cuh), vector
// form.  A warp takes up to 32 consecutive chunks: every lane reads one chunk's
// pointers and dense row address, so that a chunk costs a shuffle instead of a
// chain of dependent loads, and the entries of all of them are one contiguous
// stream.
//   Local CSR chunks run through the row-major schedule's stream (RowStream),
//   whose finished sums are added to Y instead of stored.
//   Remote CSC chunks (a few entries each: a column's rows in one partition)
//   load the dense rows of UNROLL chunks at once and scatter each to its rows;
//   a lane's features are 16 bytes of FP32, so a row's reductions are whole
//   sectors for BF16 rows too (a lane's 8 BF16 features are 32 bytes of Y).
// What bounds it: the reductions into Y in L2 (16-byte red.global.add, 4 bytes a
// feature for every remote entry).
#pragma once
#include "spmm_rows.cuh"

namespace cola {
namespace dev {

// Address of the dense row of remote chunk c of part d.
template <typename T>
__device__ __forceinline__ const T *remote_row(const PartDesc &d, const T *X, const int64_t ldx, const int64_t c)
{
    if (d.r_mode == kRemoteFromX)
        return X + (d.x_remote0 + __ldg(d.r_col + c)) * ldx;
    const int64_t w = c - d.r_begin;
    if (d.r_mode == kRemoteStagedChunk)
        return static_cast<const T *>(d.stage) + w * d.ld_stage;
    int64_t peer_off = 0;
    if (!(c >= d.local_col_lb && c < d.local_col_ub)) {
        const int peer = (__ldg(d.r_col + c) / d.npp) % d.gs + d.group_offset;
        peer_off = (int64_t)(peer - d.peid) * d.pe_stride;
    }
    return static_cast<const T *>(d.stage) + peer_off + __ldg(d.idx_ppl + w) * d.ld_stage;
}

// Local chunks [c0, c0 + n) of part d, n <= 32.
template <typename RS>
__device__ __forceinline__ void fused_local(RS &rs, const PartDesc &d, const int64_t c0, const int n, EntryBatch &eb)
{
    const int lane = rs.lane;
    int lb = 0, hb = 0, row = 0;
    if (lane < n) {
        lb = __ldg(d.l_ptr + c0 + lane);
        hb = __ldg(d.l_ptr + c0 + lane + 1);
        row = __ldg(d.l_row + c0 + lane);
    }
    const int e0 = __shfl_sync(kFull, lb, 0), e1 = __shfl_sync(kFull, hb, n - 1);
    const bool some = hb > lb;
    int mc = 0;
    float mv = 0.f;
    auto fetch = [&](int e) {
        if (e + lane < e1) {
            mc = __ldcs(d.l_col + e + lane);
            mv = __ldcs(d.l_val + e + lane);
        }
    };
    fetch(e0);
    rs.clear();
    // rows of the chunks that have entries, in the order in which they end
    const unsigned nonempty = __ballot_sync(kFull, some);
    __syncwarp();
    if (some)
        eb.row[__popc(nonempty & ((1u << lane) - 1u))] = row;
    const int32_t *rows = eb.row;
    for (int e = e0; e < e1; e += 32) {
        const unsigned mark = some && hb > e && hb <= e + 32 ? 1u << (hb - 1 - e) : 0u;
        const unsigned ends = __reduce_or_sync(kFull, mark);
        __syncwarp();
        eb.col[lane] = mc;
        eb.val[lane] = make_float2(mv, mv);
        __syncwarp();
        if (e + 32 < e1)
            fetch(e + 32);
        rs.batch(eb, rows, min(32, e1 - e), ends);
        rows += __popc(ends);
    }
}

// Remote chunks [c0, c0 + n) of part d, n <= 32; Y: row 0 of the partition.
template <typename TR, int LG, int NV, int UNROLL>
__device__ __forceinline__ void fused_remote(const PartDesc &d, const int64_t c0, const int n,
                                             const typename ElemOf<TR>::T *__restrict__ X, const int64_t ldx,
                                             float *__restrict__ Y, const int64_t ldy, const int K, const int k0,
                                             const int lane, EntryBatch &eb)
{
    using T = typename ElemOf<TR>::T;
    using TS = typename ScatterOf<TR>::type;
    constexpr int E = TS::E, NQ = NV * TR::E / E, G = 32 / LG;
    const int g = lane / LG, gl = lane % LG;
    const int koff = k0 + gl * E;
    int lb = 0, hb = 0;
    const T *src = X;
    if (lane < n) {
        lb = __ldg(d.r_ptr + c0 + lane);
        hb = __ldg(d.r_ptr + c0 + lane + 1);
        src = remote_row(d, X, ldx, c0 + lane);
    }
    const int e1 = __shfl_sync(kFull, hb, n - 1);
    int bb = __shfl_sync(kFull, lb, 0);  // entries [bb, bb + 32) are staged, the 32 after them in registers
    int mr = 0;
    float mv = 0.f;
    auto fetch = [&](int e) {
        if (e + lane < e1) {
            mr = __ldcs(d.r_row + e + lane);
            mv = __ldcs(d.r_val + e + lane);
        }
    };
    auto stage = [&]() {
        __syncwarp();
        eb.row[lane] = mr;
        eb.col[lane] = __float_as_int(mv);
        __syncwarp();
        fetch(bb + 32);
    };
    fetch(bb);
    stage();
#pragma unroll 1
    for (int q = 0; q < n; q += UNROLL) {
        typename TS::raw_t xr[UNROLL][NQ];
#pragma unroll
        for (int u = 0; u < UNROLL; u++) {
            const T *p = reinterpret_cast<const T *>(
                __shfl_sync(kFull, reinterpret_cast<unsigned long long>(src), (q + u) & 31));
#pragma unroll
            for (int j = 0; j < NQ; j++)
                if (q + u < n && koff + j * LG * E < K)
                    xr[u][j] = TS::load(p + koff + j * LG * E);
        }
#pragma unroll
        for (int u = 0; u < UNROLL; u++) {
            if (q + u >= n)
                break;
            float xs[NQ][E];
#pragma unroll
            for (int j = 0; j < NQ; j++)
                TS::unpack(xr[u][j], xs[j]);
            int s = __shfl_sync(kFull, lb, q + u);
            const int h = __shfl_sync(kFull, hb, q + u);
            while (s < h) {
                const int lim = min(h, bb + 32);
                auto add = [&](const int r, const float v) {
                    float *yp = Y + (int64_t)r * ldy + koff;
#pragma unroll
                    for (int j = 0; j < NQ; j++)
                        if (koff + j * LG * E < K) {
                            float a[E];
#pragma unroll
                            for (int i = 0; i < E; i++)
                                a[i] = v * xs[j][i];
                            red_add<E, true>(yp + j * LG * E, a);
                        }
                };
                // four entries a group read before the first is added: the
                // reductions need not wait for one another's operands
                for (; s + 3 * G + G <= lim; s += 4 * G) {
                    int r[4];
                    float v[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        r[i] = eb.row[s + i * G + g - bb];
                        v[i] = __int_as_float(eb.col[s + i * G + g - bb]);
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        add(r[i], v[i]);
                }
                for (; s < lim; s += G)
                    if (s + g < lim)
                        add(eb.row[s + g - bb], __int_as_float(eb.col[s + g - bb]));
                s = lim;
                if (lim == bb + 32) {
                    bb += 32;
                    stage();
                }
            }
        }
    }
}

// Items [0, total) over all parts as in fused_spmm_kernel, `span` consecutive
// ones (at most 32) a warp.
template <typename TR, int LG, int NV, int UNROLL, int MINB>
__global__ void __launch_bounds__(kThreads, MINB) fused_stream_kernel(const PartDesc *__restrict__ parts,
                                                                const __grid_constant__ PartDesc single, int nparts,
                                                                int64_t total, int span,
                                                                const typename ElemOf<TR>::T *__restrict__ X,
                                                                int64_t ldx, float *__restrict__ Y, int64_t ldy, int K)
{
    __shared__ EntryBatch s_ent[kWarpsPerBlock];
    pdl_launch_dependents();
    pdl_wait();
    EntryBatch &eb = s_ent[threadIdx.x >> 5];
    const int k0 = blockIdx.y * (LG * NV * TR::E);
    const int64_t w = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    const int64_t end = min(total, (w + 1) * span);
    int pidx = 0;
    for (int64_t it = w * span; it < end;) {
        const PartDesc &d = parts ? *find_part(parts, nparts, it, pidx) : single;
        const int64_t li = it - d.item0;
        int n;
        float *Yd = Y + d.y_row0 * ldy;
        if (li < d.l_num) {
            n = (int)min(end - it, d.l_num - li);
            RowStream<TR, float, LG, NV, UNROLL, true, true> rs;
            rs.init(X + d.x_local0 * ldx, ldx, Yd, ldy, K, k0, 1);
            fused_local(rs, d, d.l_begin + li, n, eb);
        } else {
            n = (int)min(end - it, (int64_t)d.l_num + d.r_num - li);
            fused_remote<TR, LG, NV, UNROLL>(d, d.r_begin + (li - d.l_num), n, X, ldx, Yd, ldy, K, k0, lane_id(), eb);
        }
        it += n;
    }
}

}  // namespace dev
}  // namespace cola
