// Fused attention aggregation over a sparsity pattern (sm_100a):
//
//     s_ij  = beta * <A_i, B_j>                 for every stored (i, j)          (the SDDMM)
//     a_ij  = softmax_j(s_ij)  or  s_ij                                           (edge softmax, optional)
//     out_i = sum_j a_ij * V_j        (V = B in the forward pass)                 (the SpMM)
//
// in ONE pass over the pattern: every gathered row B_j is used for its score and for the
// aggregation while it sits in registers, the per-edge values never reach memory, and the
// softmax is the running-maximum ("online") form, so a row needs no second sweep.  This is the
// AGNN propagation (A = B = the projected node features) without the two edge-array round trips
// and with half the gathers of SDDMM followed by SpMM.  With a separate aggregation operand V
// (template flag SEP: a second gather per entry) the same pass gives the layer's backward products
// from recomputed scores: sum_j a_ij G_j for an upstream gradient G, again without an edge array.
//
// Work unit = segment (CSR row or PCSR row piece); a group of LPR lanes owns one segment, lane gl
// holds the slice [(cf*LPR + gl)*4, +4) of A_i and of the accumulator.  Entries are taken BS at a
// time: BS gathers (128-bit loads), BS lane-partial dot products, a recursive-halving exchange
// after which lane e holds the complete score of entry e (about one shuffle per entry), one
// max / exp / sum step for the batch, then BS broadcasts of the weights and the FMAs.
//
// A row that is a single segment is normalised and stored directly.  Pieces of a split row leave
// (running max, running sum, unnormalised accumulator) in caller-provided scratch and are merged
// by agnn_combine_kernel; long rows of an unsplit layout are cut by the kernel itself when scratch is
// given (agnn_long_rows) and merged by agnn_combine_long_kernel.  Rows that no segment covers are zeroed by a memset of the output
// (split layouts only; in plain CSR every row is a segment and stores its own zeros).
#include <math_constants.h>

#include "pspmm_common.cuh"
#include "vec_ops.cuh"

namespace {

struct AgnnArgs {
    const int32_t *segPtr;
    const int32_t *target_row;  // nullptr: row == segment
    const int32_t *colIdx;
    const float *A;
    const float *B;
    const float *Vm;  // aggregated rows (SEP kernels); row stride ldV, 0 = one row shared by all columns
    float *out;
    float *scratch;  // [n_seg][4 + dim_pad] partials of split rows: max, sum, 2 unused, accumulator
    int64_t n_seg;
    int64_t ldA, ldB, ldV, ldOut;
    int32_t dim, dim_pad;
    float beta;
    int32_t softmax;
    int32_t long_row;    // unsplit rows with more entries are dealt to the first long_ctas CTAs (INT32_MAX: none are)
    int32_t long_range;  // entries per range of those CTAs
    uint32_t long_ctas;
};

// Running state of one lane group: maximum and sum of the softmax (per group), the lane's slices of
// the unnormalised accumulator.
template <int CF, int VW>
struct AgnnState {
    float m, l, acc[CF][VW];
};

// The entries [lb, hb) of one row for one lane group.  Every lane of the warp calls this together;
// `maxlen` is the longest of the warp's ranges and a group without work passes lb == hb.
template <int LPR, int CF, int BS, int VW, bool SEP>
__device__ __forceinline__ void agnn_entries(const AgnnArgs &a, const FVec<VW> (&av)[CF], const bool (&act)[CF],
                                             const int (&voff)[CF], int lb, int hb, int maxlen, int gl,
                                             AgnnState<CF, VW> &state)
{
    float m = state.m, l = state.l;
    float (&acc)[CF][VW] = state.acc;
    const int len = hb - lb;
    const int sub = gl % BS;  // position inside the batch this lane answers for

    // Column indices are read LPR at a time (lane gl <-> entry gl of the chunk, one coalesced
    // load) and one chunk ahead, so that their latency is not part of the per-batch chain.
    int c_next = (lb + gl < hb) ? __ldg(a.colIdx + lb + gl) : 0;
    for (int off0 = 0; off0 < maxlen; off0 += LPR) {
        const int c_chunk = c_next;
        {
            const int kn = lb + off0 + LPR + gl;
            c_next = (kn < hb) ? __ldg(a.colIdx + kn) : 0;
        }
#pragma unroll
        for (int b = 0; b < LPR / BS; ++b) {
            const int off = off0 + b * BS;
            if (off >= maxlen)
                break;  // warp-uniform
            const bool mine = (lb + off + sub) < hb;
            const bool full = (off + BS <= len);
            FVec<VW> x[BS][CF];
            FVec<VW> y[SEP ? BS : 1][SEP ? CF : 1];  // the rows that are aggregated, when they are not B's
            float part[BS];
            int ce[BS];
#pragma unroll
            for (int e = 0; e < BS; ++e)
                ce[e] = __shfl_sync(PSPMM_FULL_MASK, c_chunk, b * BS + e, LPR);
#pragma unroll
            for (int e = 0; e < BS; ++e) {
                const float *brow = a.B + (int64_t)ce[e] * a.ldB;
                if (full) {
#pragma unroll
                    for (int cf = 0; cf < CF; ++cf)
                        x[e][cf] = ldg_vec<VW>(brow + voff[cf]);
                } else {
                    const bool on = (off + e) < len;
#pragma unroll
                    for (int cf = 0; cf < CF; ++cf)
                        x[e][cf] = ldg_vec_if<VW>(brow + voff[cf], on);
                }
                if constexpr (SEP) {
                    const float *vrow = a.Vm + (int64_t)ce[e] * a.ldV;
                    const bool on = (off + e) < len;
#pragma unroll
                    for (int cf = 0; cf < CF; ++cf)
                        y[e][cf] = ldg_vec_if<VW>(vrow + voff[cf], on);
                }
            }
#pragma unroll
            for (int e = 0; e < BS; ++e) {
                float s = 0.f;
#pragma unroll
                for (int cf = 0; cf < CF; ++cf)
                    if (act[cf]) {
#pragma unroll
                        for (int i = 0; i < VW; ++i)
                            s = fmaf(av[cf].v[i], x[e][cf].v[i], s);
                    }
                part[e] = s;
            }
            const float score = a.beta * group_transpose_reduce<LPR, BS>(part, gl);  // entry `sub`
            float p;
            if (a.softmax) {
                float bm = mine ? score : -CUDART_INF_F;
#pragma unroll
                for (int d = BS / 2; d >= 1; d >>= 1)
                    bm = fmaxf(bm, __shfl_xor_sync(PSPMM_FULL_MASK, bm, d));
                const float m_new = fmaxf(m, bm);
                // a group past the end of its segment sees only -inf: keep its state untouched
                const bool any = m_new > -CUDART_INF_F;
                const float sc = any ? expf(m - m_new) : 1.f;
                p = (mine && any) ? expf(score - m_new) : 0.f;
                float ls = p;
#pragma unroll
                for (int d = BS / 2; d >= 1; d >>= 1)
                    ls += __shfl_xor_sync(PSPMM_FULL_MASK, ls, d);
                l = l * sc + ls;
                m = m_new;
#pragma unroll
                for (int cf = 0; cf < CF; ++cf)
#pragma unroll
                    for (int i = 0; i < VW; ++i)
                        acc[cf][i] *= sc;
            } else {
                p = mine ? score : 0.f;
            }
#pragma unroll
            for (int e = 0; e < BS; ++e) {
                const float pe = __shfl_sync(PSPMM_FULL_MASK, p, e, BS);
#pragma unroll
                for (int cf = 0; cf < CF; ++cf)
#pragma unroll
                    for (int i = 0; i < VW; ++i) {
                        if constexpr (SEP)
                            acc[cf][i] = fmaf(pe, y[e][cf].v[i], acc[cf][i]);
                        else
                            acc[cf][i] = fmaf(pe, x[e][cf].v[i], acc[cf][i]);
                    }
            }
        }
    }
    state.m = m;
    state.l = l;
}

template <int LPR, int CF, int VW>
__device__ __forceinline__ void agnn_load_row(const AgnnArgs &a, int64_t row, bool live, int gl, FVec<VW> (&av)[CF],
                                              bool (&act)[CF], int (&voff)[CF], AgnnState<CF, VW> &state)
{
    const int nvec = a.dim / VW;
#pragma unroll
    for (int cf = 0; cf < CF; ++cf) {
        const int v = cf * LPR + gl;
        act[cf] = v < nvec;
        voff[cf] = act[cf] ? v * VW : 0;
        av[cf] = (live && act[cf]) ? ldg_vec<VW>(a.A + row * a.ldA + voff[cf]) : zero_vec<VW>();
#pragma unroll
        for (int i = 0; i < VW; ++i)
            state.acc[cf][i] = 0.f;
    }
    state.m = -CUDART_INF_F;
    state.l = 0.f;
}

// Scratch slot of the piece of a long row that starts at entry p (counted from the first entry) of
// range p / long_range: rows that start in the same stretch of long_row entries are not both long,
// and only one row continues into a range, so (stretch, continues or starts) names a piece.
__device__ __forceinline__ int64_t long_piece_slot(const AgnnArgs &a, int64_t p, bool starts)
{
    return 2 * (p / a.long_row) + (starts ? 1 : 0);
}

// The first `long_ctas` CTAs look after the long rows of an unsplit layout (more than a.long_row
// entries), which the lane groups of the others pass over: one group walks a row's batches one after
// the other, so a hub row of 8 K entries held a 900 K-entry graph at dim 32 for 0.8 ms of a 20 us
// pass.  CTA c owns the entries [c, c+1) * a.long_range, finds the long rows among them, deals each
// one's entries to its lane groups, merges their states in shared memory and leaves one partial
// result per piece in scratch for agnn_combine_long_kernel.
template <int LPR, int CF, int BS, int VW, bool SEP>
__device__ __forceinline__ void agnn_long_rows(const AgnnArgs &a)
{
    constexpr int GROUPS = 256 / LPR;
    extern __shared__ float part[];  // [8][dim_pad + 2]
    const int pitch = a.dim_pad + 2;
    __shared__ int row_list[PSPMM_LONG_PER_RANGE];
    __shared__ int row_ends[2];
    __shared__ int n_long;
    const int g = threadIdx.x / LPR, gl = threadIdx.x % LPR;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t begin = __ldg(a.segPtr), end = __ldg(a.segPtr + a.n_seg);
    for (int64_t s = begin + (int64_t)blockIdx.x * a.long_range; s < end; s += (int64_t)a.long_ctas * a.long_range) {
        const int64_t e1 = s + a.long_range < end ? s + a.long_range : end;
        if (threadIdx.x == 0)
            n_long = 0;
        if (warp < 2) {
            const int r = find_segment(a.segPtr, a.n_seg, begin, end, warp == 0 ? s : e1 - 1, lane);
            if (lane == 0)
                row_ends[warp] = r;
        }
        __syncthreads();
        for (int64_t r = row_ends[0] + threadIdx.x; r <= row_ends[1]; r += 256)
            if (__ldg(a.segPtr + r + 1) - __ldg(a.segPtr + r) > a.long_row)
                row_list[atomicAdd(&n_long, 1)] = (int)r;
        __syncthreads();
        for (int i = 0; i < n_long; ++i) {
            const int r = row_list[i];
            const int64_t rb = __ldg(a.segPtr + r), re = __ldg(a.segPtr + r + 1);
            const int64_t lo = rb > s ? rb : s, hi = re < e1 ? re : e1;
            const int share = (int)((hi - lo + GROUPS - 1) / GROUPS);
            int64_t b = lo + (int64_t)g * share;
            b = b < hi ? b : hi;
            const int64_t e = b + share < hi ? b + share : hi;
            FVec<VW> av[CF];
            bool act[CF];
            int voff[CF];
            AgnnState<CF, VW> st;
            agnn_load_row<LPR, CF, VW>(a, r, true, gl, av, act, voff, st);
            agnn_entries<LPR, CF, BS, VW, SEP>(a, av, act, voff, (int)b, (int)e, share, gl, st);
            // the lane groups of a warp merge by shuffles, the warps in shared memory
            float M = st.m;
#pragma unroll
            for (int d = LPR; d < 32; d <<= 1)
                M = fmaxf(M, __shfl_xor_sync(PSPMM_FULL_MASK, M, d));
            const float w = !a.softmax ? 1.f : (st.m > -CUDART_INF_F ? expf(st.m - M) : 0.f);
            float *mine = part + warp * pitch;
            float L = st.l * w;
#pragma unroll
            for (int d = LPR; d < 32; d <<= 1)
                L += __shfl_xor_sync(PSPMM_FULL_MASK, L, d);
            if (lane == 0) {
                mine[0] = M;
                mine[1] = L;
            }
#pragma unroll
            for (int cf = 0; cf < CF; ++cf)
#pragma unroll
                for (int j = 0; j < VW; ++j) {
                    float x = st.acc[cf][j] * w;
#pragma unroll
                    for (int d = LPR; d < 32; d <<= 1)
                        x += __shfl_xor_sync(PSPMM_FULL_MASK, x, d);
                    if (lane < LPR && act[cf])
                        mine[2 + voff[cf] + j] = x;
                }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 8; ++q)
                M = fmaxf(M, part[q * pitch]);
            float *ps = a.scratch + long_piece_slot(a, lo - begin, rb >= s) * (int64_t)(4 + a.dim_pad);
            for (int j = (int)threadIdx.x - 1; j < a.dim; j += 256) {  // (thread 0 starts with the sum of the weights)
                float t = 0.f;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float mq = part[q * pitch];
                    const float wq = !a.softmax ? 1.f : (mq > -CUDART_INF_F ? expf(mq - M) : 0.f);
                    t = fmaf(wq, part[q * pitch + 2 + j], t);  // (column -1 is the warp's sum)
                }
                if (j < 0) {
                    ps[0] = M;
                    ps[1] = t;
                } else {
                    ps[4 + j] = t;
                }
            }
            __syncthreads();
        }
        __syncthreads();
    }
}

template <int LPR, int CF, int BS, int VW, bool SEP = false>
__global__ void __launch_bounds__(256) agnn_fused_kernel(const AgnnArgs a)
{
    static_assert(BS <= LPR, "a batch cannot be wider than the lane group");
    pdl_launch_dependents();
    if (blockIdx.x < a.long_ctas) {
        agnn_long_rows<LPR, CF, BS, VW, SEP>(a);
        return;
    }
    const int gpc = blockDim.x / LPR;
    const int g = threadIdx.x / LPR;
    const int gl = threadIdx.x % LPR;
    const int64_t seg = (int64_t)(blockIdx.x - a.long_ctas) * gpc + g;
    // Lanes of dead groups run along with empty ranges: the shuffles below are full-warp.
    bool live = seg < a.n_seg;
    int lb = 0, hb = 0;
    int64_t row = 0;
    bool single = true;
    if (live) {
        lb = __ldg(a.segPtr + seg);
        hb = __ldg(a.segPtr + seg + 1);
        row = seg;
        if (a.target_row) {
            const int me = __ldg(a.target_row + seg);
            const int prev = seg > 0 ? __ldg(a.target_row + seg - 1) : -1;
            const int next = seg + 1 < a.n_seg ? __ldg(a.target_row + seg + 1) : -1;
            row = me;
            single = (prev != me) && (next != me);
        } else if (hb - lb > a.long_row) {
            live = false;
            hb = lb;
        }
    }
    FVec<VW> av[CF];
    bool act[CF];
    int voff[CF];
    AgnnState<CF, VW> st;
    agnn_load_row<LPR, CF, VW>(a, row, live, gl, av, act, voff, st);
    int maxlen = hb - lb;
    if constexpr (LPR < 32)
        maxlen = __reduce_max_sync(PSPMM_FULL_MASK, maxlen);
    agnn_entries<LPR, CF, BS, VW, SEP>(a, av, act, voff, lb, hb, maxlen, gl, st);
    if (!live)
        return;
    if (single) {
        const float inv = a.softmax ? (st.l > 0.f ? 1.f / st.l : 0.f) : 1.f;
        float *orow = a.out + row * a.ldOut;
#pragma unroll
        for (int cf = 0; cf < CF; ++cf)
            if (act[cf]) {
                float v[VW];
#pragma unroll
                for (int i = 0; i < VW; ++i)
                    v[i] = st.acc[cf][i] * inv;
                st_stream_vec<VW>(orow + voff[cf], v);
            }
    } else {
        float *ps = a.scratch + seg * (int64_t)(4 + a.dim_pad);
        if (gl == 0) {
            ps[0] = st.m;
            ps[1] = st.l;
        }
#pragma unroll
        for (int cf = 0; cf < CF; ++cf)
            if (act[cf])
                st_vec<VW>(ps + 4 + voff[cf], st.acc[cf]);
    }
}

// Merges the `count` pieces of one row; slot(t) is where piece t lies.  All `warps` warps of a team
// (the caller's warp alone, or the whole CTA with red != nullptr) take pieces in turn, four of them
// in flight per lane; a lane carries four columns, and a CTA adds the warps' sums in shared memory.
// (One warp walking all pieces of a row took 0.54 ms for a hub row of 900 pieces.)
template <typename Slot>
__device__ __forceinline__ void merge_pieces(const AgnnArgs &a, int64_t row, int64_t count, const Slot &slot, int warp,
                                             int warps, int lane, float *red)
{
    const int64_t stride = 4 + a.dim_pad;
    float M = -CUDART_INF_F;
    if (a.softmax) {
        for (int64_t t = lane; t < count; t += 32)
            M = fmaxf(M, a.scratch[slot(t) * stride]);
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1)
            M = fmaxf(M, __shfl_xor_sync(PSPMM_FULL_MASK, M, d));
    }
    float L = 0.f;
    float acc[2][4] = {};
    for (int64_t t0 = warp * 4; t0 < count; t0 += warps * 4) {
        float w[4];
        const float *ps[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool on = t0 + u < count;
            ps[u] = a.scratch + slot(on ? t0 + u : t0) * stride;
            w[u] = 1.f;
            if (a.softmax && on) {
                const float mt = ps[u][0];
                w[u] = mt > -CUDART_INF_F ? expf(mt - M) : 0.f;
                L += w[u] * ps[u][1];
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = (h * 32 + lane) * 4;
            if (j < a.dim) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (t0 + u >= count)
                        break;
                    const float4 x = *reinterpret_cast<const float4 *>(ps[u] + 4 + j);
                    acc[h][0] = fmaf(w[u], x.x, acc[h][0]);
                    acc[h][1] = fmaf(w[u], x.y, acc[h][1]);
                    acc[h][2] = fmaf(w[u], x.z, acc[h][2]);
                    acc[h][3] = fmaf(w[u], x.w, acc[h][3]);
                }
            }
        }
    }
    if (red) {
        float *mine = red + warp * (256 + 1);
        if (lane == 0)
            mine[256] = L;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                mine[(h * 32 + lane) * 4 + i] = acc[h][i];
        __syncthreads();
        float *orow = a.out + row * a.ldOut;
        for (int j = warp * 32 + lane; j < a.dim; j += warps * 32) {
            float s = 0.f, l = 0.f;
            for (int q = 0; q < warps; ++q) {
                s += red[q * 257 + j];
                l += red[q * 257 + 256];
            }
            orow[j] = a.softmax ? (l > 0.f ? s / l : 0.f) : s;
        }
        __syncthreads();
        return;
    }
    const float inv = a.softmax ? (L > 0.f ? 1.f / L : 0.f) : 1.f;
    float *orow = a.out + row * a.ldOut;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int j = (h * 32 + lane) * 4;
        if (j < a.dim)
            *reinterpret_cast<float4 *>(orow + j) =
                make_float4(acc[h][0] * inv, acc[h][1] * inv, acc[h][2] * inv, acc[h][3] * inv);
    }
}

// A CTA looks at MERGE_SPAN segments (or rows) and merges the rows whose first piece lies there: a
// warp per row up to MERGE_WARP pieces, the whole CTA for the others.
constexpr int MERGE_SPAN = 64;
constexpr int MERGE_WARP = 32;

__global__ void __launch_bounds__(256) agnn_combine_kernel(const AgnnArgs a)
{
    __shared__ float red[8 * 257];
    __shared__ int list[MERGE_SPAN];
    __shared__ int n_list;
    if (threadIdx.x == 0)
        n_list = 0;
    __syncthreads();
    pdl_wait();
    const int64_t s = (int64_t)blockIdx.x * MERGE_SPAN + threadIdx.x;
    if (threadIdx.x < MERGE_SPAN && s + 1 < a.n_seg) {
        const int me = __ldg(a.target_row + s);
        if (__ldg(a.target_row + s + 1) == me && (s == 0 || __ldg(a.target_row + s - 1) != me))
            list[atomicAdd(&n_list, 1)] = (int)s;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = n_list;
    for (int i = warp; i < n; i += 8) {
        const int64_t seg = list[i];
        const int me = __ldg(a.target_row + seg);
        const bool in = seg + lane < a.n_seg && __ldg(a.target_row + seg + lane) == me;
        const int count = __popc(__ballot_sync(PSPMM_FULL_MASK, in));
        static_assert(MERGE_WARP == 32, "the ballot counts up to 32 pieces");
        const bool more = seg + 32 < a.n_seg && __ldg(a.target_row + seg + 32) == me;
        if (!more) {
            merge_pieces(a, me, count, [&](int64_t t) { return seg + t; }, 0, 1, lane, nullptr);
            if (lane == 0)
                list[i] = -1;
        }
    }
    __syncthreads();
    for (int i = 0; i < n; ++i) {
        const int64_t seg = list[i];
        if (seg < 0)
            continue;
        const int me = __ldg(a.target_row + seg);
        int64_t count = 0;
        while (true) {
            const int64_t t = seg + count + threadIdx.x;
            const int c = __syncthreads_count(t < a.n_seg && __ldg(a.target_row + t) == me);
            count += c;
            if (c < 256)
                break;
        }
        merge_pieces(a, me, count, [&](int64_t t) { return seg + t; }, warp, 8, lane, red);
    }
}

__global__ void __launch_bounds__(256) agnn_combine_long_kernel(const AgnnArgs a)
{
    __shared__ float red[8 * 257];
    __shared__ int list[MERGE_SPAN];
    __shared__ int n_list;
    if (threadIdx.x == 0)
        n_list = 0;
    __syncthreads();
    const int64_t r0 = (int64_t)blockIdx.x * MERGE_SPAN + threadIdx.x;
    if (threadIdx.x < MERGE_SPAN && r0 < a.n_seg && __ldg(a.segPtr + r0 + 1) - __ldg(a.segPtr + r0) > a.long_row)
        list[atomicAdd(&n_list, 1)] = (int)r0;
    __syncthreads();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = n_list;
    const int64_t begin = __ldg(a.segPtr);
    for (int pass = 0; pass < 2; ++pass) {
        // first the rows a warp can merge, then the long ones
        for (int i = pass ? 0 : warp; i < n; i += pass ? 1 : 8) {
            const int64_t row = list[i];
            const int64_t rb = __ldg(a.segPtr + row) - begin, re = __ldg(a.segPtr + row + 1) - begin;
            const int64_t c0 = rb / a.long_range;
            const int64_t count = (re - 1) / a.long_range - c0 + 1;
            if ((count > MERGE_WARP) != (pass == 1))
                continue;
            const auto slot = [&](int64_t t) {
                return t == 0 ? long_piece_slot(a, rb, true) : long_piece_slot(a, (c0 + t) * a.long_range, false);
            };
            merge_pieces(a, row, count, slot, pass ? warp : 0, pass ? 8 : 1, lane, pass ? red : nullptr);
        }
    }
}

template <int LPR, int CF, int BS, int VW, bool SEP = false>
void launch_fused(const AgnnArgs &a, cudaStream_t st)
{
    const int gpc = 256 / LPR;
    const int64_t gx = (a.n_seg + gpc - 1) / gpc + a.long_ctas;
    agnn_fused_kernel<LPR, CF, BS, VW, SEP><<<(unsigned)gx, 256, a.long_ctas ? 8 * (a.dim_pad + 2) * 4 : 0, st>>>(a);
}

}  // namespace

extern "C" int pspmm_agnn_scratch_bytes(int64_t n_seg, int32_t dim, size_t *bytes)
{
    if (n_seg < 0 || dim <= 0 || !bytes)
        return PSPMM_E_ARG;
    const int64_t dim_pad = (dim + 3) / 4 * 4;
    *bytes = (size_t)n_seg * (size_t)(4 + dim_pad) * sizeof(float);
    return PSPMM_OK;
}

// Entries above which a row of an unsplit layout is cut, and the bytes its pieces may need.
static int agnn_long_row(int64_t nnz) { return pspmm_long_row_threshold(nnz); }

extern "C" int pspmm_agnn_long_scratch_bytes(int64_t nnz, int32_t dim, size_t *bytes)
{
    if (nnz < 0 || dim <= 0 || !bytes)
        return PSPMM_E_ARG;
    const int t = agnn_long_row(nnz);
    const int64_t slots = t == INT32_MAX ? 0 : 2 * ((nnz + t - 1) / t);
    *bytes = (size_t)slots * (size_t)(4 + (dim + 3) / 4 * 4) * sizeof(float);
    return PSPMM_OK;
}

extern "C" int pspmm_agnn_fused_csr(const int32_t *rowPtr, const int32_t *colIdx, const float *A,
                                    const float *B, float *out, int64_t n_rows, int64_t nnz, int32_t dim,
                                    int64_t ldA, int64_t ldB, int64_t ldOut, float beta, int32_t softmax,
                                    int32_t vec_width, int32_t lanes_per_row, int32_t batch,
                                    const int32_t *rowPtr_split, const int32_t *target_row,
                                    int64_t n_seg, void *scratch, size_t scratch_bytes, void *stream)
{
    return pspmm_agnn_fused_apply_csr(rowPtr, colIdx, A, B, B, out, n_rows, nnz, dim, ldA, ldB, ldB, ldOut, beta,
                                      softmax, vec_width, lanes_per_row, batch, rowPtr_split, target_row, n_seg,
                                      scratch, scratch_bytes, stream);
}

extern "C" int pspmm_agnn_fused_apply_csr(const int32_t *rowPtr, const int32_t *colIdx, const float *A,
                                          const float *B, const float *V, float *out, int64_t n_rows, int64_t nnz,
                                          int32_t dim, int64_t ldA, int64_t ldB, int64_t ldV, int64_t ldOut,
                                          float beta, int32_t softmax, int32_t vec_width, int32_t lanes_per_row,
                                          int32_t batch, const int32_t *rowPtr_split, const int32_t *target_row,
                                          int64_t n_seg, void *scratch, size_t scratch_bytes, void *stream)
{
    if (n_rows < 0 || nnz < 0 || dim <= 0)
        return PSPMM_E_ARG;
    if (!V || (ldV != 0 && ldV < dim))
        return PSPMM_E_ARG;
    const bool sep = (V != B) || (ldV != ldB);
    if (sep && (ldV % 4 != 0 || ((uintptr_t)V) % 16 != 0))
        return PSPMM_E_UNSUPPORTED;
    if (n_rows >= INT32_MAX || nnz > INT32_MAX)
        return PSPMM_E_RANGE;
    const bool split = target_row != nullptr || rowPtr_split != nullptr;
    if (split && (!rowPtr_split || !target_row || n_seg < 0 || n_seg >= INT32_MAX))
        return PSPMM_E_ARG;
    if (!split && !rowPtr)
        return PSPMM_E_ARG;
    if (!A || !B || !out || ldA < dim || ldB < dim || ldOut < dim)
        return PSPMM_E_ARG;
    if (nnz > 0 && !colIdx)
        return PSPMM_E_ARG;
    if (batch != 0 && batch != 4 && batch != 8 && batch != 16)
        return PSPMM_E_CONFIG;
    if (lanes_per_row != 0 && lanes_per_row != 4 && lanes_per_row != 8 && lanes_per_row != 16 && lanes_per_row != 32)
        return PSPMM_E_CONFIG;
    // 128-bit accesses throughout: dim a multiple of 4 (at most 256) and 16-byte aligned rows.
    if (dim % 4 != 0 || dim > 256 || ldA % 4 != 0 || ldB % 4 != 0 || ldOut % 4 != 0 ||
        ((uintptr_t)A) % 16 != 0 || ((uintptr_t)B) % 16 != 0 || ((uintptr_t)out) % 16 != 0)
        return PSPMM_E_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    if (n_rows == 0)
        return PSPMM_OK;
    AgnnArgs a;
    a.segPtr = split ? rowPtr_split : rowPtr;
    a.target_row = split ? target_row : nullptr;
    a.colIdx = colIdx;
    a.A = A;
    a.B = B;
    a.Vm = V;
    a.ldV = ldV;
    a.out = out;
    a.scratch = (float *)scratch;
    a.n_seg = split ? n_seg : n_rows;
    a.ldA = ldA;
    a.ldB = ldB;
    a.ldOut = ldOut;
    a.dim = dim;
    a.dim_pad = (dim + 3) / 4 * 4;
    a.beta = beta;
    a.softmax = softmax ? 1 : 0;
    if (split) {
        const size_t need = (size_t)n_seg * (size_t)(4 + a.dim_pad) * sizeof(float);
        if (n_seg > 0 && (!scratch || scratch_bytes < need || ((uintptr_t)scratch) % 16 != 0))
            return PSPMM_E_ARG;
        // rows without any segment stay zero
        PSPMM_CUDA_TRY(cudaMemset2DAsync(out, (size_t)ldOut * 4, 0, (size_t)dim * 4, (size_t)n_rows, st));
        if (n_seg == 0)
            return PSPMM_OK;
    }
    a.long_row = INT32_MAX;
    a.long_range = 0;
    a.long_ctas = 0;
    if (!split && scratch && ((uintptr_t)scratch) % 16 == 0) {
        size_t need = 0;
        pspmm_agnn_long_scratch_bytes(nnz, dim, &need);
        if (need > 0 && scratch_bytes >= need) {
            a.long_row = agnn_long_row(nnz);
            a.long_range = 8 * a.long_row;
            a.long_ctas = (uint32_t)((nnz + a.long_range - 1) / a.long_range);
        }
    }
    // Launch shape: floats per lane per load (VW: 8 = 256-bit loads when the rows are 32-byte
    // aligned, else 4), lanes per row (LPR), slices per lane (CF = ceil(dim / VW / LPR)) and
    // entries per batch (BS).  Few lanes per row put more entries into every warp instruction (the
    // 128-bit form at 16 lanes is bound by instruction issue); wide loads keep the L1 wavefronts
    // full (the 128-bit form at 4 lanes is bound by the L1 data pipe).  Defaults = measured best.
    // (a separate aggregation operand doubles the gathered registers: batches of 4, and with 256-bit
    // loads one slice per lane)
    const bool can8 = dim % 8 == 0 && dim >= 32 && ldA % 8 == 0 && ldB % 8 == 0 && ((uintptr_t)A) % 32 == 0 &&
                      ((uintptr_t)B) % 32 == 0 && (!sep || (ldV % 8 == 0 && ((uintptr_t)V) % 32 == 0));
    if (sep)
        batch = 4;
    if (vec_width != 0 && vec_width != 4 && vec_width != 8)
        return PSPMM_E_CONFIG;
    const int vw = (vec_width == 8 && !can8) ? 4 : (vec_width ? vec_width : (can8 ? 8 : 4));
    const int nvec = dim / vw;
    int lpr = lanes_per_row;
    if (lpr == 0)
        lpr = vw == 8 ? (nvec <= 8 ? 4 : (nvec <= 16 ? 8 : 16)) : (nvec <= 16 ? 4 : (nvec <= 32 ? 8 : 16));
    const int cf_max = vw == 8 ? 2 : 4;
    int cf = (nvec + lpr - 1) / lpr;
    while (cf > cf_max && lpr < 32) {
        lpr *= 2;
        cf = (nvec + lpr - 1) / lpr;
    }
    if (sep && lanes_per_row == 0) {  // two gathered rows per entry: at most two slices per lane (one of 32 bytes) keeps them in registers
        while (cf > (vw == 8 ? 1 : 2) && lpr < 32) {
            lpr *= 2;
            cf = (nvec + lpr - 1) / lpr;
        }
    }
    if (cf > cf_max)
        return PSPMM_E_UNSUPPORTED;
    if (cf == 3)
        cf = 4;
    int bs = batch ? batch : 4;
    if (bs > lpr)
        bs = lpr;
    if (cf * vw >= 16 && bs > 4)
        bs = 4;
    if (cf * vw >= 8 && bs > 8)
        bs = 8;
    bool ok = false;
#define AGNN_CASE_SEP(LPR_, CF_, VW_)                                 \
    if (!ok && sep && vw == VW_ && lpr == LPR_ && cf == CF_ && bs == 4) { \
        launch_fused<LPR_, CF_, 4, VW_, true>(a, st);                 \
        ok = true;                                                    \
    }
    AGNN_CASE_SEP(4, 1, 4) AGNN_CASE_SEP(4, 2, 4) AGNN_CASE_SEP(4, 4, 4) AGNN_CASE_SEP(8, 1, 4) AGNN_CASE_SEP(8, 2, 4)
    AGNN_CASE_SEP(8, 4, 4) AGNN_CASE_SEP(16, 1, 4) AGNN_CASE_SEP(16, 2, 4) AGNN_CASE_SEP(16, 4, 4)
    AGNN_CASE_SEP(32, 1, 4) AGNN_CASE_SEP(32, 2, 4)
    AGNN_CASE_SEP(4, 1, 8) AGNN_CASE_SEP(8, 1, 8) AGNN_CASE_SEP(16, 1, 8) AGNN_CASE_SEP(32, 1, 8)
    AGNN_CASE_SEP(4, 2, 8) AGNN_CASE_SEP(8, 2, 8) AGNN_CASE_SEP(16, 2, 8)
#undef AGNN_CASE_SEP
    if (sep && !ok)
        return PSPMM_E_UNSUPPORTED;
#define AGNN_CASE(LPR_, CF_, BS_, VW_)                             \
    if (!ok && vw == VW_ && lpr == LPR_ && cf == CF_ && bs == BS_) { \
        launch_fused<LPR_, CF_, BS_, VW_>(a, st);                  \
        ok = true;                                                 \
    }
    AGNN_CASE(4, 1, 4, 4) AGNN_CASE(4, 2, 4, 4) AGNN_CASE(4, 4, 4, 4)
    AGNN_CASE(8, 1, 4, 4) AGNN_CASE(8, 1, 8, 4) AGNN_CASE(8, 2, 4, 4) AGNN_CASE(8, 2, 8, 4) AGNN_CASE(8, 4, 4, 4)
    AGNN_CASE(16, 1, 4, 4) AGNN_CASE(16, 1, 8, 4) AGNN_CASE(16, 1, 16, 4) AGNN_CASE(16, 2, 4, 4) AGNN_CASE(16, 2, 8, 4)
    AGNN_CASE(16, 4, 4, 4)
    AGNN_CASE(32, 1, 4, 4) AGNN_CASE(32, 1, 8, 4) AGNN_CASE(32, 1, 16, 4) AGNN_CASE(32, 2, 4, 4) AGNN_CASE(32, 2, 8, 4)
    AGNN_CASE(4, 1, 4, 8) AGNN_CASE(4, 2, 4, 8)
    AGNN_CASE(8, 1, 4, 8) AGNN_CASE(8, 1, 8, 8) AGNN_CASE(8, 2, 4, 8)
    AGNN_CASE(16, 1, 4, 8) AGNN_CASE(16, 1, 8, 8) AGNN_CASE(16, 2, 4, 8)
    AGNN_CASE(32, 1, 4, 8) AGNN_CASE(32, 1, 8, 8)
#undef AGNN_CASE
    if (!ok)
        return PSPMM_E_UNSUPPORTED;
    PSPMM_CUDA_TRY(cudaGetLastError());
    const unsigned spans = (unsigned)((a.n_seg + MERGE_SPAN - 1) / MERGE_SPAN);
    if (split)
        PSPMM_CUDA_TRY(launch_dependent(agnn_combine_kernel, dim3(spans), 256, 0, st, a));
    else if (a.long_ctas)
        PSPMM_CUDA_TRY(launch_dependent(agnn_combine_long_kernel, dim3(spans), 256, 0, st, a));
    return PSPMM_OK;
}
