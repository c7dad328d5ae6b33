// Fused attention aggregation over a sparsity pattern (sm_100a):
//
//     s_ij  = beta * <A_i, B_j>                 for every stored (i, j)          (the SDDMM)
//     a_ij  = softmax_j(s_ij)  or  s_ij                                           (edge softmax, optional)
//     out_i = sum_j a_ij * V_j        (V = B in the forward pass)                 (the SpMM)
//
// in ONE pass over the pattern: every gathered row B_j is used for its score and for the
// aggregation while it sits in registers, the per-edge values reach memory only where a training forward
// leaves its scores, and the softmax's weights are taken against a reference that follows the largest score so far
// ("online" form), so a row needs no second sweep.  This is the
// AGNN propagation (A = B = the projected node features) without the two edge-array round trips
// and with half the gathers of SDDMM followed by SpMM.  With a separate aggregation operand V
// (template flag SEP: a second gather per entry) the same pass gives the layer's backward products
// from recomputed scores: sum_j a_ij G_j for an upstream gradient G, again without an edge array.  Where the
// forward left its scores (SCORES_LEAVE), the backward takes them and gathers G alone (SCORES_TAKE).
//
// Work unit = segment (CSR row or PCSR row piece); a group of LPR lanes owns one segment, lane gl
// holds the slice [(cf*LPR + gl)*4, +4) of A_i and of the accumulator.  Entries are taken BS at a
// time: BS gathers (128-bit loads), BS lane-partial dot products, a recursive-halving exchange
// after which lane e holds the complete score of entry e (about one shuffle per entry), one
// exp per lane (and a vote on whether the reference moves) for the batch, then BS broadcasts of the weights and the FMAs.
//
// A row that is a single segment is normalised and stored directly.  Pieces of a split row leave
// (reference, sum of weights, unnormalised accumulator) in caller-provided scratch and are merged
// by agnn_combine_kernel; long rows of an unsplit layout are cut by the kernel itself when scratch is
// given (agnn_long_kernel).  Rows that no segment covers are zeroed by a memset of the output
// (split layouts only; in plain CSR every row is a segment and stores its own zeros).
#include <math_constants.h>

#include "long_rows.cuh"
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
    float *scratch;  // [n_seg][4 + dim_pad] partials of split rows: reference, sum, 2 unused, accumulator
    int64_t n_seg;
    int64_t ldA, ldB, ldV, ldOut;
    int32_t dim, dim_pad;
    float beta;
    const float *beta_dev;  // where beta lies on the device, or nullptr: `beta`
    int32_t softmax;
    float *scores;          // scores per entry: SCORES_LEAVE kernels write them, SCORES_TAKE kernels read them
    double *col_sums;       // COL kernels: one partial sum per CTA
    int32_t n_col_sums;     // CTAs of the first kernel that own segments, then the shares of long rows
    float *col_out;
    LongArgs lng;  // unsplit layouts: how long rows are cut (totals == nullptr: they are not)
};

// What a kernel does with a.scores.
enum { SCORES_NONE, SCORES_LEAVE, SCORES_TAKE };

// Sum over the CTA's 256 threads, stored by thread 0.
__device__ __forceinline__ void cta_sum_to(double *dst, double x)
{
    __shared__ double warps[8];
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1)
        x += __shfl_xor_sync(PSPMM_FULL_MASK, x, d);
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
        warps[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w)
            t += warps[w];
        *dst = t;
    }
}

// One CTA adds up the partial sums.
__global__ void __launch_bounds__(256) agnn_col_sum_kernel(const AgnnArgs a)
{
    pdl_wait();
    double x = 0.0;
    for (int i = threadIdx.x; i < a.n_col_sums; i += 256)
        x += __ldcg(a.col_sums + i);
    double *sum = a.col_sums + a.n_col_sums;
    cta_sum_to(sum, x);
    if (threadIdx.x == 0)
        *a.col_out = (float)*sum;
}

// Running state of one lane group: maximum and sum of the softmax (per group), the lane's slices of
// the unnormalised accumulator.
// With COL also the lane's part of the sum over the row's entries of column id * <V_i, V_j> (the score
// gradient that the layer's attention weight receives), from the slices of row i in `vv`.
template <int CF, int VW, bool COL>
struct AgnnState {
    float beta;
    float m, l, acc[CF][VW];
    float t;
    FVec<VW> vv[COL ? CF : 1];
};

// The entries [lb, hb) of one row for one lane group.  Every lane of the warp calls this together;
// `maxlen` is the longest of the warp's ranges and a group without work passes lb == hb.
template <int LPR, int CF, int BS, int VW, bool SEP, bool COL, int SCORES, bool SOFTMAX>
__device__ __forceinline__ void agnn_entries(const AgnnArgs &a, const FVec<VW> (&av)[CF], const bool (&act)[CF],
                                             const int (&voff)[CF], int lb, int hb, int maxlen, int gl,
                                             AgnnState<CF, VW, COL> &state)
{
    float m = state.m, l = state.l;
    float (&acc)[CF][VW] = state.acc;
    const int len = hb - lb;
    const unsigned ub = lb, ue = hb;  // (lb and the longest range of the warp can add up to more than 2^31)
    const int sub = gl % BS;  // position inside the batch this lane answers for

    // The rows of a batch, and those that are aggregated when they are not B's.  Beyond a row's entries the 16-byte
    // forms with several slices per lane keep an earlier batch's and leave it out of the sums: clearing it took an
    // instruction per float, and that, the addresses and the loads of idle lanes were a third of all
    // (12 M entries, softmax: dim 100 584 -> 474 us, dim 148 1074 -> 867).  With one slice or 32-byte loads the
    // zeros are free (dim 128 487, without them 489; dim 32 160 and 167, dim 16 44 and 46).
    constexpr bool KEEP = VW == 4 && CF > 1;
    FVec<VW> x[BS][CF];
    FVec<VW> y[SEP ? BS : 1][SEP ? CF : 1];
    const float *laneB = a.B + gl * VW, *laneV = a.Vm + gl * VW;
    const unsigned ldB_lo = (unsigned)(a.ldB * 4), ldB_hi = (unsigned)((unsigned long long)(a.ldB * 4) >> 32);
    const unsigned ldV_lo = (unsigned)(a.ldV * 4), ldV_hi = (unsigned)((unsigned long long)(a.ldV * 4) >> 32);
    if constexpr (KEEP) {
#pragma unroll
        for (int e = 0; e < BS; ++e)
#pragma unroll
            for (int cf = 0; cf < CF; ++cf) {
                x[e][cf] = zero_vec<VW>();
                if constexpr (SEP)
                    y[e][cf] = zero_vec<VW>();
            }
    }

    // Column indices are read LPR at a time (lane gl <-> entry gl of the chunk, one coalesced
    // load) and one chunk ahead, so that their latency is not part of the per-batch chain.
    int c_next = (ub + gl < ue) ? __ldg(a.colIdx + (ub + gl)) : 0;
    for (int off0 = 0; off0 < maxlen; off0 += LPR) {
        const int c_chunk = c_next;
        {
            const unsigned kn = ub + off0 + LPR + gl;
            c_next = (kn < ue) ? __ldg(a.colIdx + kn) : 0;
        }
#pragma unroll
        for (int b = 0; b < LPR / BS; ++b) {
            const int off = off0 + b * BS;
            if (off >= maxlen)
                break;  // warp-uniform
            const bool mine = (ub + off + sub) < ue;
            float part[BS];
            int ce[BS];
#pragma unroll
            for (int e = 0; e < BS; ++e)
                ce[e] = __shfl_sync(PSPMM_FULL_MASK, c_chunk, b * BS + e, LPR);
            // Predicated, not branched on whether the batch is full: the groups of a warp are at different
            // entries of their rows, and a branch issued the loads of one after those of the others
            // (115 M entries at dim 64: 2.7 ms with the branch, 2.2 without; with two operands 5.2, 3.6).
#pragma unroll
            for (int e = 0; e < BS; ++e) {
                const bool on = (off + e) < len;
                if constexpr (KEEP) {
                    const float *brow = row_start(laneB, ce[e], ldB_lo, ldB_hi);
#pragma unroll
                    for (int cf = 0; cf < CF; ++cf)
                        ldg_vec_keep<VW>(x[e][cf], brow + cf * LPR * VW, on && act[cf]);
                    if constexpr (SEP) {
                        const float *vrow = row_start(laneV, ce[e], ldV_lo, ldV_hi);
#pragma unroll
                        for (int cf = 0; cf < CF; ++cf)
                            ldg_vec_keep<VW>(y[e][cf], vrow + cf * LPR * VW, on && act[cf]);
                    }
                } else {
                    const float *brow = a.B + (int64_t)ce[e] * a.ldB;
#pragma unroll
                    for (int cf = 0; cf < CF; ++cf)
                        x[e][cf] = ldg_vec_if<VW>(brow + voff[cf], on);
                    if constexpr (SEP) {
                        const float *vrow = a.Vm + (int64_t)ce[e] * a.ldV;
#pragma unroll
                        for (int cf = 0; cf < CF; ++cf)
                            y[e][cf] = ldg_vec_if<VW>(vrow + voff[cf], on);
                    }
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
            const float score = state.beta * group_transpose_reduce<LPR, BS>(part, gl);  // entry `sub`
            float p;
            if constexpr (SOFTMAX) {
                // m: what the exponentials are taken against, at most 8 below the largest score so far.  It moves when a
                // score exceeds it by more (a vote of the warp, mostly no), and l stays with the lanes until the end: two
                // exchanges, an exponential and the accumulator's scaling leave the chain of every batch (12 M entries, split: dim 128
                // 487 -> 468 us, 64 264 -> 250, 32 160 -> 148; moved by every larger score, 480, 256 and 153).  The weights, up to e^8, are
                // scaled by 2^-12, exactly, so that the sums have the range that weights up to 1 leave them (no time).
                const float over = score - m;
                if (__any_sync(PSPMM_FULL_MASK, mine && over > 8.f)) {
                    float bm = mine ? score : -CUDART_INF_F;
#pragma unroll
                    for (int d = BS / 2; d >= 1; d >>= 1)
                        bm = fmaxf(bm, __shfl_xor_sync(PSPMM_FULL_MASK, bm, d));
                    const float m_new = fmaxf(m, bm);
                    const float sc = m_new > -CUDART_INF_F ? expf(m - m_new) : 1.f;
                    m = m_new;
                    l *= sc;
#pragma unroll
                    for (int cf = 0; cf < CF; ++cf)
#pragma unroll
                        for (int i = 0; i < VW; ++i)
                            acc[cf][i] *= sc;
                }
                // (a group whose scores so far are all -inf keeps an empty state)
                p = mine && m > -CUDART_INF_F ? expf(score - m) * 0x1p-12f : 0.f;
                l += p;
            } else {
                p = mine ? score : 0.f;
            }
            if constexpr (SCORES == SCORES_LEAVE) {
                if (mine && gl < BS)
                    __stcs(a.scores + (ub + off + sub), score);
            }
            if constexpr (COL) {
#pragma unroll
                for (int e = 0; e < BS; ++e) {
                    float d = 0.f;
#pragma unroll
                    for (int cf = 0; cf < CF; ++cf)
                        if (act[cf]) {
#pragma unroll
                            for (int i = 0; i < VW; ++i)
                                d = fmaf(state.vv[cf].v[i], y[e][cf].v[i], d);
                        }
                    if (!KEEP || (off + e) < len)
                        state.t = fmaf((float)ce[e], d, state.t);
                }
            }
#pragma unroll
            for (int e = 0; e < BS; ++e) {
                const float pe = __shfl_sync(PSPMM_FULL_MASK, p, e, BS);
#pragma unroll
                for (int cf = 0; cf < CF; ++cf) {
                    const FVec<VW> &r = SEP ? y[SEP ? e : 0][SEP ? cf : 0] : x[e][cf];
                    if constexpr (KEEP) {
                        fma_vec_if<VW>(acc[cf], pe, r.v, (off + e) < len);
                    } else {
#pragma unroll
                        for (int i = 0; i < VW; ++i)
                            acc[cf][i] = fmaf(pe, r.v[i], acc[cf][i]);
                    }
                }
            }
        }
    }
    state.m = m;
    state.l = l;
}

// The group's sum of the weights that its lanes hold.
template <int BS>
__device__ __forceinline__ float agnn_weight_sum(float l, unsigned lanes)
{
#pragma unroll
    for (int d = BS / 2; d >= 1; d >>= 1)
        l += __shfl_xor_sync(lanes, l, d);
    return l;
}

// The same for scores that lie in a.scores: one gather per entry (the rows of a.Vm) and no exchange.  A training
// step's backward pass takes the forward's: 115 M entries, dim 64: 3.64 ms with the scores recomputed from a
// second gather, 1.72 (17 TB/s of gathered rows; the bare gather takes 1.4); the forward writes them in 0.09 ms of 1.89.
// Bound: the latency of eight 32-byte loads in flight per lane at two resident CTAs.
template <int LPR, int CF, int BS, int VW, bool COL>
__device__ __forceinline__ void agnn_scored_entries(const AgnnArgs &a, const bool (&act)[CF], const int (&voff)[CF], int lb,
                                                    int hb, int maxlen, int gl, AgnnState<CF, VW, COL> &state)
{
    const int len = hb - lb;
    const unsigned ub = lb, ue = hb;
    int c_next = 0;
    float p_next = 0.f;
    auto fetch = [&](unsigned k) {  // lane gl <-> entry gl of a chunk, one chunk ahead
        c_next = k < ue ? __ldg(a.colIdx + k) : 0;
        p_next = k < ue ? __ldcs(a.scores + k) : 0.f;
    };
    fetch(ub + gl);
    for (int off0 = 0; off0 < maxlen; off0 += LPR) {
        const int c_chunk = c_next;
        const float p_chunk = p_next;
        fetch(ub + off0 + LPR + gl);
#pragma unroll
        for (int b = 0; b < LPR / BS; ++b) {
            const int off = off0 + b * BS;
            if (off >= maxlen)
                break;  // warp-uniform
            FVec<VW> y[BS][CF];
            float pe[BS];
            int ce[BS];
#pragma unroll
            for (int e = 0; e < BS; ++e) {
                ce[e] = __shfl_sync(PSPMM_FULL_MASK, c_chunk, b * BS + e, LPR);
                pe[e] = __shfl_sync(PSPMM_FULL_MASK, p_chunk, b * BS + e, LPR);
            }
#pragma unroll
            for (int e = 0; e < BS; ++e) {
                const float *vrow = a.Vm + (int64_t)ce[e] * a.ldV;
#pragma unroll
                for (int cf = 0; cf < CF; ++cf)
                    y[e][cf] = ldg_vec_if<VW>(vrow + voff[cf], (off + e) < len);
            }
#pragma unroll
            for (int e = 0; e < BS; ++e) {
                if constexpr (COL) {
                    float d = 0.f;
#pragma unroll
                    for (int cf = 0; cf < CF; ++cf)
                        if (act[cf]) {
#pragma unroll
                            for (int i = 0; i < VW; ++i)
                                d = fmaf(state.vv[cf].v[i], y[e][cf].v[i], d);
                        }
                    state.t = fmaf((float)ce[e], d, state.t);
                }
#pragma unroll
                for (int cf = 0; cf < CF; ++cf)
#pragma unroll
                    for (int i = 0; i < VW; ++i)
                        state.acc[cf][i] = fmaf(pe[e], y[e][cf].v[i], state.acc[cf][i]);
            }
        }
    }
}

template <int LPR, int CF, int VW, bool COL, int SCORES>
__device__ __forceinline__ void agnn_load_row(const AgnnArgs &a, int64_t row, bool live, int gl, FVec<VW> (&av)[CF],
                                              bool (&act)[CF], int (&voff)[CF], AgnnState<CF, VW, COL> &state)
{
    const int nvec = a.dim / VW;
#pragma unroll
    for (int cf = 0; cf < CF; ++cf) {
        const int v = cf * LPR + gl;
        act[cf] = v < nvec;
        voff[cf] = act[cf] ? v * VW : 0;
        if constexpr (SCORES != SCORES_TAKE)
            av[cf] = (live && act[cf]) ? ldg_vec<VW>(a.A + row * a.ldA + voff[cf]) : zero_vec<VW>();
        if constexpr (COL)
            state.vv[cf] = (live && act[cf]) ? ldg_vec<VW>(a.Vm + row * a.ldV + voff[cf]) : zero_vec<VW>();
#pragma unroll
        for (int i = 0; i < VW; ++i)
            state.acc[cf][i] = 0.f;
    }
    state.m = -CUDART_INF_F;
    state.l = 0.f;
}

// Resident CTAs the register budget is cut for: 16 floats of a row per lane would otherwise take 142
// registers and leave one (12 M entries at dim 128: 1,040 us instead of 570).  Taking scores, three CTAs of 80 registers
// and eight rows in flight beat two of 128 up to 16 lanes (steps of 4 M entries, dim 128 677 -> 640 us, 12 M 1011 -> 970; 115 M,
// dim 64: the kernel 1.77 -> 1.72 ms); on 32 lanes they spill, and the long rows' kernel, with more state, loses 3 %.
template <int CF, int VW, bool SEP>
struct AgnnOcc {
    static constexpr int MIN_CTAS = SEP ? (CF * VW >= 16 ? 1 : 2) : (CF * VW >= 16 ? 2 : 3);
};

template <int LPR, int CF, int BS, int VW, bool SEP, bool COL, int SCORES, bool SOFTMAX>
__global__ void __launch_bounds__(256, SCORES == SCORES_TAKE && LPR <= 16 ? 3 : AgnnOcc<CF, VW, SEP>::MIN_CTAS) agnn_fused_kernel(const AgnnArgs a)
{
    static_assert(BS <= LPR, "a batch cannot be wider than the lane group");
    pdl_launch_dependents();
    if (blockIdx.x < (unsigned)a.lng.scan_ctas) {
        long_scan(a.lng, a.segPtr, a.n_seg, blockIdx.x);
        return;
    }
    const int gpc = blockDim.x / LPR;
    const int g = threadIdx.x / LPR;
    const int gl = threadIdx.x % LPR;
    const int64_t seg = (int64_t)(blockIdx.x - a.lng.scan_ctas) * gpc + g;
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
        } else if (a.lng.totals && hb - lb > PSPMM_LONG_ROW) {  // agnn_long_kernel takes it
            live = false;
            hb = lb;
        }
    }
    FVec<VW> av[CF];
    bool act[CF];
    int voff[CF];
    AgnnState<CF, VW, COL> st;
    st.beta = a.beta_dev ? __ldg(a.beta_dev) : a.beta;
    st.t = 0.f;
    agnn_load_row<LPR, CF, VW, COL, SCORES>(a, row, live, gl, av, act, voff, st);
    int maxlen = hb - lb;
    if constexpr (LPR < 32)
        maxlen = __reduce_max_sync(PSPMM_FULL_MASK, maxlen);
    if constexpr (SCORES == SCORES_TAKE)
        agnn_scored_entries<LPR, CF, BS, VW, COL>(a, act, voff, lb, hb, maxlen, gl, st);
    else
        agnn_entries<LPR, CF, BS, VW, SEP, COL, SCORES, SOFTMAX>(a, av, act, voff, lb, hb, maxlen, gl, st);
    if constexpr (COL)
        cta_sum_to(a.col_sums + (blockIdx.x - a.lng.scan_ctas), (double)st.t);
    if constexpr (SOFTMAX)
        st.l = agnn_weight_sum<BS>(st.l, PSPMM_FULL_MASK);
    if (!live)
        return;
    if (single) {
        const float inv = SOFTMAX ? (st.l > 0.f ? 1.f / st.l : 0.f) : 1.f;
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

// The long rows of an unsplit layout (long_rows.cuh): one lane group walks a row's batches one after the
// other, so a hub row of 8 K entries held a 900 K-entry graph at dim 32 for 0.8 ms of a 20 us pass.
// The entries of a share are dealt to the lane groups in equal spans; a group's states (maximum, sum,
// accumulator) at the ends of its span and the shares' states of a row meet in shared memory and in
// scratch as the pieces of a split row do.
template <int LPR, int CF, int BS, int VW, bool SEP, bool COL, int SCORES, bool SOFTMAX>
__global__ void __launch_bounds__(256, AgnnOcc<CF, VW, SEP>::MIN_CTAS) agnn_long_kernel(const AgnnArgs a)
{
    constexpr int G = 256 / LPR;
    constexpr int STEP = 64;  // entries per group between two looks at the row ends of a warp
    extern __shared__ float parts[];  // [G][first or last piece][reference, sum, dim_pad columns]
    __shared__ LongShare::Shared sh;
    const int pitch = a.dim_pad + 2;
    const int g = threadIdx.x / LPR, gl = threadIdx.x % LPR;
    const int share = blockIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    double t_sum = 0.0;
    LongShare job;
    const bool any = job.begin(a.lng, sh, share);
    const int64_t stride = 4 + a.dim_pad;
    while (any && job.look(sh, a.segPtr, a.n_seg)) {
        const int total = job.total;
        if (total == 0)
            continue;
        const int span = (total + G - 1) / G;
        const int start = g * span;
        const int stop = start + span < total ? start + span : total;
        int p = start;
        int i = p < stop ? job.row_of(sh, p) : 0;
        FVec<VW> av[CF];
        bool act[CF];
        int voff[CF];
        AgnnState<CF, VW, COL> st;
        st.beta = a.beta_dev ? __ldg(a.beta_dev) : a.beta;
        st.t = 0.f;
        agnn_load_row<LPR, CF, VW, COL, SCORES>(a, sh.row[i], p < stop, gl, av, act, voff, st);
        bool from_row_start = p < stop && p == job.off(sh, i);
        while (__any_sync(PSPMM_FULL_MASK, p < stop)) {
            int lb = 0, count = 0, row_end = 0;
            if (p < stop) {
                row_end = job.off(sh, i + 1);
                const int row_stop = row_end < stop ? row_end : stop;
                count = row_stop - p < STEP ? row_stop - p : STEP;
                lb = sh.lo[i] - job.off(sh, i) + p;
            }
            const int longest = LPR < 32 ? __reduce_max_sync(PSPMM_FULL_MASK, count) : count;
            if constexpr (SCORES == SCORES_TAKE)
                agnn_scored_entries<LPR, CF, BS, VW, COL>(a, act, voff, lb, lb + count, longest, gl, st);
            else
                agnn_entries<LPR, CF, BS, VW, SEP, COL, SCORES, SOFTMAX>(a, av, act, voff, lb, lb + count, longest, gl, st);
            if (count == 0)
                continue;
            p += count;
            if (p != stop && p != row_end)
                continue;
            if constexpr (COL) {
                t_sum += (double)st.t;
                st.t = 0.f;
            }
            // a piece is complete: all of the row in this share, or the first or last piece of the span
            if constexpr (SOFTMAX)
                st.l = agnn_weight_sum<BS>(st.l, LPR == 32 ? PSPMM_FULL_MASK : ((1u << LPR) - 1u) << ((threadIdx.x & 31) / LPR * LPR));
            int s0, s1;
            job.shares_of(sh, i, s0, s1);
            if (from_row_start && p == row_end && s0 == s1) {
                const float inv = SOFTMAX ? (st.l > 0.f ? 1.f / st.l : 0.f) : 1.f;
                float *orow = a.out + (int64_t)sh.row[i] * a.ldOut;
#pragma unroll
                for (int cf = 0; cf < CF; ++cf)
                    if (act[cf]) {
                        float v[VW];
#pragma unroll
                        for (int j = 0; j < VW; ++j)
                            v[j] = st.acc[cf][j] * inv;
                        st_stream_vec<VW>(orow + voff[cf], v);
                    }
            } else {
                float *mine = parts + (g * 2 + (job.off(sh, i) <= start ? 0 : 1)) * pitch;
                if (gl == 0) {
                    mine[0] = st.m;
                    mine[1] = st.l;
                }
#pragma unroll
                for (int cf = 0; cf < CF; ++cf)
                    if (act[cf]) {
#pragma unroll
                        for (int j = 0; j < VW; ++j)
                            mine[2 + voff[cf] + j] = st.acc[cf][j];
                    }
            }
            ++i;
            from_row_start = true;
            agnn_load_row<LPR, CF, VW, COL, SCORES>(a, p < stop ? sh.row[i] : 0, p < stop, gl, av, act, voff, st);
        }
        __syncthreads();
        // Rows that several groups or shares hold: their pieces of this share, in order.
        const int row0 = sh.edge[0], rows = sh.edge[1] - row0 + 1;
        const int each = a.dim + 1;  // (column -1 is the sum of the weights)
        for (int t = threadIdx.x; t < rows * each; t += 256) {
            const int i2 = row0 + t / each, j = t % each - 1;
            const int off0 = job.off(sh, i2);
            const int g0 = off0 / span, g1 = (job.off(sh, i2 + 1) - 1) / span;
            int s0, s1;
            job.shares_of(sh, i2, s0, s1);
            if (g0 == g1 && s0 == s1)
                continue;
            float M = -CUDART_INF_F, sum = 0.f, l = 0.f;
            for (int q = g0; q <= g1; ++q)
                M = fmaxf(M, parts[(q * 2 + (off0 <= q * span ? 0 : 1)) * pitch]);
            for (int q = g0; q <= g1; ++q) {
                const float *ps = parts + (q * 2 + (off0 <= q * span ? 0 : 1)) * pitch;
                const float w = !SOFTMAX ? 1.f : (ps[0] > -CUDART_INF_F ? expf(ps[0] - M) : 0.f);
                sum = fmaf(w, ps[2 + j], sum);
                l = fmaf(w, ps[1], l);
            }
            if (s0 != s1) {
                float *out = a.lng.partials + LongShare::slot(share, s0) * stride;
                if (j < 0) {
                    out[0] = M;
                    out[1] = sum;
                } else {
                    out[4 + j] = sum;
                }
            } else if (j >= 0) {
                a.out[(int64_t)sh.row[i2] * a.ldOut + j] = !SOFTMAX ? sum : (l > 0.f ? sum / l : 0.f);
            }
        }
        job.arrive(a.lng, sh, 0, 1);
        for (int q = 0; q < 2; ++q) {
            if (!sh.last[q])
                continue;
            int s0, s1;
            job.shares_of(sh, sh.edge[q], s0, s1);
            for (int j = threadIdx.x; j < a.dim; j += 256) {
                float M = -CUDART_INF_F, sum = 0.f, l = 0.f;
                for (int c = s0; c <= s1; ++c)
                    M = fmaxf(M, __ldcg(a.lng.partials + LongShare::slot(c, s0) * stride));
                for (int c = s0; c <= s1; ++c) {
                    const float *ps = a.lng.partials + LongShare::slot(c, s0) * stride;
                    const float m = __ldcg(ps);
                    const float w = !SOFTMAX ? 1.f : (m > -CUDART_INF_F ? expf(m - M) : 0.f);
                    sum = fmaf(w, __ldcg(ps + 4 + j), sum);
                    l = fmaf(w, __ldcg(ps + 1), l);
                }
                a.out[(int64_t)sh.row[sh.edge[q]] * a.ldOut + j] = !SOFTMAX ? sum : (l > 0.f ? sum / l : 0.f);
            }
        }
        __syncthreads();
    }
    if constexpr (COL)
        cta_sum_to(a.col_sums + a.n_col_sums - a.lng.shares + share, t_sum);
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

template <int LPR, int CF, int BS, int VW, bool SEP, bool COL, int SCORES, bool SOFTMAX>
void launch_form(const AgnnArgs &a, cudaStream_t st)
{
    const int gpc = 256 / LPR;
    const int64_t gx = (a.n_seg + gpc - 1) / gpc + a.lng.scan_ctas;
    agnn_fused_kernel<LPR, CF, BS, VW, SEP, COL, SCORES, SOFTMAX><<<(unsigned)gx, 256, 0, st>>>(a);
    if (a.lng.totals)
        launch_dependent(agnn_long_kernel<LPR, CF, BS, VW, SEP, COL, SCORES, SOFTMAX>, dim3((unsigned)a.lng.shares), 256,
                         gpc * 2 * (a.dim_pad + 2) * 4, st, a);
}

template <int LPR, int CF, int BS, int VW, bool SEP = false, bool COL = false, int SCORES = SCORES_NONE>
void launch_fused(const AgnnArgs &a, cudaStream_t st)
{
    if constexpr (!COL && SCORES == SCORES_NONE) {
        if (a.softmax) {
            launch_form<LPR, CF, BS, VW, SEP, COL, SCORES, true>(a, st);
            return;
        }
    }
    launch_form<LPR, CF, BS, VW, SEP, COL, SCORES, false>(a, st);  // (the layers' passes have no softmax)
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

// Long rows' shares: two CTAs of agnn_long_kernel per SM.
static void agnn_long_layout(LongArgs *a, int64_t n_rows, int64_t nnz)
{
    long_layout(a, n_rows, nnz, pspmm_sm_count(), 2, 1);
}
static size_t agnn_long_bytes(const LongArgs &a, int32_t dim)
{
    return long_head_bytes(a) + (size_t)a.shares * 2 * (4 + (dim + 3) / 4 * 4) * sizeof(float);
}

extern "C" int pspmm_agnn_long_scratch_bytes(int64_t n_rows, int64_t nnz, int32_t dim, size_t *bytes)
{
    if (n_rows < 0 || nnz < 0 || dim <= 0 || !bytes)
        return PSPMM_E_ARG;
    *bytes = 0;
    if (nnz > PSPMM_LONG_ROW && n_rows > 0) {
        LongArgs a;
        agnn_long_layout(&a, n_rows, nnz);
        *bytes = agnn_long_bytes(a, dim);
    }
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

// Partial sums of the column-weighted scores: a CTA of 4 lanes per segment at the least, and the shares.
static size_t agnn_sums_bytes(int64_t n_seg)
{
    LongArgs a;
    long_layout(&a, n_seg, 0, pspmm_sm_count(), 2 * 16, 1);  // (at most 16 waves of shares)
    return (size_t)((n_seg + 7) / 8 + a.shares + 2) * sizeof(double);
}

// What the entry points share.  beta_dev: beta on the device (nullptr: the value); col_out: where the sum
// over all entries of column id * <V_i, V_j> goes (nullptr: it is not formed), with `sums` of
// agnn_col_sums(...) + 1 doubles for it.
static int agnn_run(const int32_t *rowPtr, const int32_t *colIdx, const float *A, const float *B, const float *V,
                    float *out, int64_t n_rows, int64_t nnz, int32_t dim, int64_t ldA, int64_t ldB, int64_t ldV,
                    int64_t ldOut, float beta, const float *beta_dev, int32_t softmax, int32_t vec_width,
                    int32_t lanes_per_row, int32_t batch, const int32_t *rowPtr_split, const int32_t *target_row,
                    int64_t n_seg, void *scratch, size_t scratch_bytes, float *col_out, double *sums, size_t sums_bytes,
                    float *scores, bool take_scores, void *stream)
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
    if (split && (!rowPtr_split || (n_seg > 0 && !target_row) || n_seg < 0 || n_seg >= INT32_MAX))
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
    if (col_out && (n_rows == 0 || (split && n_seg == 0)))
        PSPMM_CUDA_TRY(cudaMemsetAsync(col_out, 0, sizeof(float), st));
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
    a.beta_dev = beta_dev;
    a.scores = scores;
    a.col_sums = sums;
    a.n_col_sums = 0;
    a.col_out = col_out;
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
    a.lng = LongArgs{};
    if (!split && scratch && ((uintptr_t)scratch) % 16 == 0 && nnz > PSPMM_LONG_ROW) {
        agnn_long_layout(&a.lng, n_rows, nnz);
        if (long_fits(a.lng, nnz) && scratch_bytes >= agnn_long_bytes(a.lng, dim))
            long_place(&a.lng, scratch);
        else
            a.lng = LongArgs{};
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
    if ((sep || take_scores) && lanes_per_row == 0) {  // two gathered rows per entry: at most two slices per lane (one of 32 bytes) keeps them in registers
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
    // (the column-weighted sum is built for the shapes that the rules above choose)
    const int64_t sum_ctas = (a.n_seg + 256 / lpr - 1) / (256 / lpr);
    if (col_out) {
        a.n_col_sums = (int32_t)(sum_ctas + a.lng.shares);
        if (!sums || sums_bytes < (size_t)(a.n_col_sums + 1) * sizeof(double))
            return PSPMM_E_ARG;
    }
#define AGNN_CASE_TAKE(LPR_, CF_, VW_)                                                   \
    if (!ok && take_scores && vw == VW_ && lpr == LPR_ && cf == CF_) {                   \
        if (col_out)                                                                     \
            launch_fused<LPR_, CF_, LPR_ < 8 ? 4 : 8, VW_, true, true, SCORES_TAKE>(a, st);  \
        else                                                                             \
            launch_fused<LPR_, CF_, LPR_ < 8 ? 4 : 8, VW_, true, false, SCORES_TAKE>(a, st); \
        ok = true;                                                                       \
    }
    AGNN_CASE_TAKE(4, 1, 4) AGNN_CASE_TAKE(4, 2, 4) AGNN_CASE_TAKE(8, 2, 4) AGNN_CASE_TAKE(16, 2, 4) AGNN_CASE_TAKE(32, 2, 4)
    AGNN_CASE_TAKE(4, 1, 8) AGNN_CASE_TAKE(8, 1, 8) AGNN_CASE_TAKE(16, 1, 8) AGNN_CASE_TAKE(32, 1, 8)
#undef AGNN_CASE_TAKE
#define AGNN_CASE_LEAVE(LPR_, CF_, VW_)                                          \
    if (!ok && scores && vw == VW_ && lpr == LPR_ && cf == CF_) {                \
        launch_fused<LPR_, CF_, 4, VW_, false, false, SCORES_LEAVE>(a, st);      \
        ok = true;                                                               \
    }
    AGNN_CASE_LEAVE(4, 1, 4) AGNN_CASE_LEAVE(4, 2, 4) AGNN_CASE_LEAVE(4, 4, 4) AGNN_CASE_LEAVE(8, 4, 4) AGNN_CASE_LEAVE(16, 4, 4)
    AGNN_CASE_LEAVE(4, 1, 8) AGNN_CASE_LEAVE(4, 2, 8) AGNN_CASE_LEAVE(8, 2, 8) AGNN_CASE_LEAVE(16, 2, 8)
#undef AGNN_CASE_LEAVE
    if (scores && !ok)
        return PSPMM_E_UNSUPPORTED;
#define AGNN_CASE_COL(LPR_, CF_, VW_)                                          \
    if (!ok && sep && col_out && vw == VW_ && lpr == LPR_ && cf == CF_) {      \
        launch_fused<LPR_, CF_, 4, VW_, true, true>(a, st);                    \
        ok = true;                                                             \
    }
    AGNN_CASE_COL(4, 1, 4) AGNN_CASE_COL(4, 2, 4) AGNN_CASE_COL(8, 2, 4) AGNN_CASE_COL(16, 2, 4) AGNN_CASE_COL(32, 2, 4)
    AGNN_CASE_COL(4, 1, 8) AGNN_CASE_COL(8, 1, 8) AGNN_CASE_COL(16, 1, 8) AGNN_CASE_COL(32, 1, 8)
#undef AGNN_CASE_COL
    if (col_out && !ok)
        return PSPMM_E_UNSUPPORTED;
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
    if (split)
        PSPMM_CUDA_TRY(launch_dependent(agnn_combine_kernel, dim3((unsigned)((a.n_seg + MERGE_SPAN - 1) / MERGE_SPAN)),
                                        256, 0, st, a));
    if (col_out)
        PSPMM_CUDA_TRY(launch_dependent(agnn_col_sum_kernel, dim3(1), 256, 0, st, a));
    return PSPMM_OK;
}

extern "C" int pspmm_agnn_fused_apply_csr(const int32_t *rowPtr, const int32_t *colIdx, const float *A,
                                          const float *B, const float *V, float *out, int64_t n_rows, int64_t nnz,
                                          int32_t dim, int64_t ldA, int64_t ldB, int64_t ldV, int64_t ldOut,
                                          float beta, int32_t softmax, int32_t vec_width, int32_t lanes_per_row,
                                          int32_t batch, const int32_t *rowPtr_split, const int32_t *target_row,
                                          int64_t n_seg, void *scratch, size_t scratch_bytes, void *stream)
{
    return agnn_run(rowPtr, colIdx, A, B, V, out, n_rows, nnz, dim, ldA, ldB, ldV, ldOut, beta, nullptr, softmax,
                    vec_width, lanes_per_row, batch, rowPtr_split, target_row, n_seg, scratch, scratch_bytes, nullptr,
                    nullptr, 0, nullptr, false, stream);
}

extern "C" int pspmm_agnn_layer_scratch_bytes(int64_t n_rows, int64_t nnz, int64_t n_seg, int32_t dim, size_t *bytes)
{
    if (n_rows < 0 || nnz < 0 || n_seg < 0 || dim <= 0 || !bytes)
        return PSPMM_E_ARG;
    size_t own = 0;
    int rc = n_seg > 0 ? pspmm_agnn_scratch_bytes(n_seg, dim, &own) : pspmm_agnn_long_scratch_bytes(n_rows, nnz, dim, &own);
    if (rc)
        return rc;
    *bytes = (own + 255) / 256 * 256 + agnn_sums_bytes(n_seg > 0 ? n_seg : n_rows);
    return PSPMM_OK;
}

extern "C" int pspmm_agnn_layer_forward(const int32_t *rowPtr, const int32_t *colIdx, const float *X, float *out,
                                        int64_t n_rows, int64_t nnz, int32_t dim, int64_t ldX, int64_t ldOut,
                                        const float *beta, const int32_t *rowPtr_split, const int32_t *target_row,
                                        int64_t n_seg, void *scratch, size_t scratch_bytes, void *stream)
{
    return pspmm_agnn_layer_forward_scores(rowPtr, colIdx, X, out, nullptr, n_rows, nnz, dim, ldX, ldOut, beta, rowPtr_split,
                                           target_row, n_seg, scratch, scratch_bytes, stream);
}

extern "C" int pspmm_agnn_layer_forward_scores(const int32_t *rowPtr, const int32_t *colIdx, const float *X, float *out,
                                               float *scores, int64_t n_rows, int64_t nnz, int32_t dim, int64_t ldX,
                                               int64_t ldOut, const float *beta, const int32_t *rowPtr_split,
                                               const int32_t *target_row, int64_t n_seg, void *scratch,
                                               size_t scratch_bytes, void *stream)
{
    if (!beta)
        return PSPMM_E_ARG;
    return agnn_run(rowPtr, colIdx, X, X, X, out, n_rows, nnz, dim, ldX, ldX, ldX, ldOut, 0.f, beta, 0, 0, 0, 0,
                    rowPtr_split, target_row, n_seg, scratch, scratch_bytes, nullptr, nullptr, 0, scores, false, stream);
}

// What the two backward passes share: the scores are recomputed from X, or taken.
static int agnn_backward(const int32_t *rowPtr, const int32_t *colIdx, const float *X, const float *scores, const float *G,
                         float *D, float *d_beta, int64_t n_rows, int64_t nnz, int32_t dim, int64_t ldX, int64_t ldG,
                         int64_t ldD, const float *beta, const int32_t *rowPtr_split, const int32_t *target_row,
                         int64_t n_seg, void *scratch, size_t scratch_bytes, void *stream)
{
    size_t need = 0;
    int rc = pspmm_agnn_layer_scratch_bytes(n_rows, nnz, rowPtr_split ? n_seg : 0, dim, &need);
    if (rc)
        return rc;
    if (!scratch || scratch_bytes < need || (uintptr_t)scratch % 16 != 0)
        return PSPMM_E_ARG;
    const size_t sums = agnn_sums_bytes(rowPtr_split ? n_seg : n_rows), own = need - sums;
    return agnn_run(rowPtr, colIdx, X, X, G, D, n_rows, nnz, dim, ldX, ldX, ldG, ldD, 0.f, beta, 0, 0, 0, 4,
                    rowPtr_split, target_row, n_seg, own ? scratch : nullptr, own, d_beta,
                    (double *)((char *)scratch + own), sums, const_cast<float *>(scores), scores != nullptr, stream);
}

extern "C" int pspmm_agnn_layer_backward(const int32_t *rowPtr, const int32_t *colIdx, const float *X, const float *G,
                                         float *D, float *d_beta, int64_t n_rows, int64_t nnz, int32_t dim, int64_t ldX,
                                         int64_t ldG, int64_t ldD, const float *beta, const int32_t *rowPtr_split,
                                         const int32_t *target_row, int64_t n_seg, void *scratch, size_t scratch_bytes,
                                         void *stream)
{
    if (!beta || !G)
        return PSPMM_E_ARG;
    return agnn_backward(rowPtr, colIdx, X, nullptr, G, D, d_beta, n_rows, nnz, dim, ldX, ldG, ldD, beta, rowPtr_split,
                         target_row, n_seg, scratch, scratch_bytes, stream);
}

extern "C" int pspmm_agnn_layer_backward_scores(const int32_t *rowPtr, const int32_t *colIdx, const float *scores,
                                                const float *G, float *D, float *d_beta, int64_t n_rows, int64_t nnz,
                                                int32_t dim, int64_t ldG, int64_t ldD, const int32_t *rowPtr_split,
                                                const int32_t *target_row, int64_t n_seg, void *scratch,
                                                size_t scratch_bytes, void *stream)
{
    if (!G || (nnz > 0 && !scores))
        return PSPMM_E_ARG;
    // (the operands of the scores are not read: G stands in for them in what the passes check)
    static const float none = 0.f;
    return agnn_backward(rowPtr, colIdx, G, scores ? scores : &none, G, D, d_beta, n_rows, nnz, dim, ldG, ldG, ldD, nullptr,
                         rowPtr_split, target_row, n_seg, scratch, scratch_bytes, stream);
}
