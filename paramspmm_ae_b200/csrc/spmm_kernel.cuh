// Segment SpMM kernel for sm_100a.
//
// Work unit: a "segment" = one CSR row, one PCSR row piece, or the V x 1 block-row forms of
// either.  A group of LPR lanes (LPR = 2..32, a power of two, so 32/LPR groups share a warp)
// owns `rows_per_group` CONSECUTIVE segments, whose entries are therefore one contiguous
// range of colIdx / val.  Lane gl of the group covers the dense columns
// [(cf*LPR + gl)*VW, +VW) for cf = 0..CF-1, so one group-wide load reads LPR*VW*4 contiguous
// bytes of a row of B (128-bit loads for VW = 4).
//
// Staging: the group first copies its segment pointers (and, for split layouts, the target
// rows of its segments and of the two neighbouring ones) into shared memory, then streams its
// entry range through a small shared-memory window (CAP entries, column index and value
// interleaved).  All lanes of a group need the same (column, value) pair for an entry; they
// get it with one broadcast LDS.64 instead of two register shuffles, which halves the
// load/store-unit wavefronts spent on distributing A, and the pointer -> entries -> gather
// dependency is paid once per group of rows instead of once per row.  Groups synchronise only
// among their own lanes, so groups of one warp walk rows of different lengths independently.
//
// Inner loop per entry and lane: LDS.64, one IMAD.WIDE, CF x LDG.128, 4*CF FFMA.  The gathers
// of U consecutive entries are issued before their FMAs (U*CF independent 16-byte loads in
// flight per lane); row tails fall through batches of U/2, U/4, ... 1 entries.  Lanes beyond
// the last dense column (dim not a multiple of LPR*VW) read column 0 of the same row instead
// of being predicated, and simply do not store.
//
// Output: consecutive segments of one group that target the same row are summed in
// registers.  A row whose segments all lie inside one group is stored with streaming stores
// (rows without entries store zeros, so the output needs no prior memset).  A row that
// straddles groups receives one vector RED per lane from each of them; such rows are zeroed
// beforehand by zero_shared_rows_kernel (pspmm_api.cu).  In a split layout rows that no
// segment covers lie between the target rows of consecutive segments: every group zeroes the
// short gap that follows each of its rows (up to PSPMM_GAP_MAX rows); longer gaps are left to
// the pre-pass.
//
// Long rows of an unsplit layout are left to spmm_long_rows_kernel below, which cuts them over the
// whole GPU; here they are passed over.
#pragma once

#include <type_traits>

#include "long_rows.cuh"
#include "pspmm_common.cuh"
#include "vec_ops.cuh"

template <int LPR, int V>
struct SpmmTile {
    static constexpr int CAP = (LPR * 4 < 16) ? 16 : ((LPR * 4 > 64) ? 64 : LPR * 4);
    // Per-group shared memory: pointers [RPG_MAX+1], target rows [RPG_MAX+2] (padded to a
    // multiple of 8 bytes), then CAP entries of (1 + V) words.
    static constexpr int HEAD_WORDS = ((PSPMM_RPG_MAX + 1) + (PSPMM_RPG_MAX + 2) + 1) / 2 * 2;
    static constexpr int GROUP_WORDS = HEAD_WORDS + CAP * (1 + V);
};

// One batch of UU entries starting at shared-memory index e: gathers first, FMAs after.  PACK takes two columns per
// multiply-add: the long rows' kernel gains 3 - 7 % (R-MAT of 16 M entries unsplit, 32 columns: 478 -> 454 us; power
// law of 2.5 M 67.6 -> 62.8), the segment kernel loses as much: its register budgets have no room for pairs.
template <int UU, int LPR, int VW, int CF, int V, bool PACK>
__device__ __forceinline__ void spmm_batch(const int *ent, int e, const char *const (&bcol)[CF],
                                           unsigned ldB_bytes, unsigned long long keep,
                                           float (&acc)[V][CF][VW])
{
    int c[UU];
    float v[UU][V];
#pragma unroll
    for (int u = 0; u < UU; ++u) {
        if constexpr (V == 1) {
            const int2 cv = *reinterpret_cast<const int2 *>(ent + 2 * (e + u));
            c[u] = cv.x;
            v[u][0] = __int_as_float(cv.y);
        } else {
            c[u] = ent[(1 + V) * (e + u)];
#pragma unroll
            for (int w = 0; w < V; ++w)
                v[u][w] = __int_as_float(ent[(1 + V) * (e + u) + 1 + w]);
        }
    }
    FVec<VW> x[UU][CF];
#pragma unroll
    for (int u = 0; u < UU; ++u)
#pragma unroll
        for (int cf = 0; cf < CF; ++cf)
            x[u][cf] = ldg_vec_hint<VW>(row_slice(bcol[cf], c[u], ldB_bytes), keep);
#pragma unroll
    for (int u = 0; u < UU; ++u)
#pragma unroll
        for (int w = 0; w < V; ++w) {
            // Block layouts carry explicit zeros for absent lanes; they are skipped, as the
            // reference does, so a non-finite B entry cannot leak through them.
            if (V > 1 && v[u][w] == 0.f)
                continue;
#pragma unroll
            for (int cf = 0; cf < CF; ++cf) {
                if constexpr (PACK) {
                    fma_vec<VW>(acc[w][cf], v[u][w], x[u][cf].v);
                } else {
#pragma unroll
                    for (int i = 0; i < VW; ++i)
                        acc[w][cf][i] = fmaf(v[u][w], x[u][cf].v[i], acc[w][cf][i]);
                }
            }
        }
}

// Entries [e, eh) of the staged window: batches of U, the tail in halves of it.
template <int U, int LPR, int VW, int CF, int V, bool PACK = false>
__device__ __forceinline__ void spmm_entries(const int *ent, int e, int eh, const char *const (&bcol)[CF],
                                             unsigned ldB_bytes, unsigned long long keep, float (&acc)[V][CF][VW])
{
    for (; e + U <= eh; e += U)
        spmm_batch<U, LPR, VW, CF, V, PACK>(ent, e, bcol, ldB_bytes, keep, acc);
    if constexpr (U >= 16) {
        if (e + 8 <= eh) {
            spmm_batch<8, LPR, VW, CF, V, PACK>(ent, e, bcol, ldB_bytes, keep, acc);
            e += 8;
        }
    }
    if constexpr (U >= 8) {
        if (e + 4 <= eh) {
            spmm_batch<4, LPR, VW, CF, V, PACK>(ent, e, bcol, ldB_bytes, keep, acc);
            e += 4;
        }
    }
    if constexpr (U >= 4) {
        if (e + 2 <= eh) {
            spmm_batch<2, LPR, VW, CF, V, PACK>(ent, e, bcol, ldB_bytes, keep, acc);
            e += 2;
        }
    }
    if constexpr (U >= 2) {
        if (e < eh)
            spmm_batch<1, LPR, VW, CF, V, PACK>(ent, e, bcol, ldB_bytes, keep, acc);
    }
}

// Copies entries [k, k + fill) into a group's window, column and value(s) side by side.
template <int LPR, int V>
__device__ __forceinline__ void spmm_stage(const SpmmArgs &a, int *ent, int k0, int fill, int gl, unsigned long long stream)
{
    for (int i = gl; i < fill; i += LPR) {
        const int k = k0 + i;
        if constexpr (V == 1) {
            // (no value array: the pattern itself, every stored entry counts as 1)
            *reinterpret_cast<int2 *>(ent + 2 * i) =
                make_int2(ldg_stream_b32(a.colIdx + k, stream),
                          a.val ? ldg_stream_b32(a.val + k, stream) : __float_as_int(1.f));
        } else {
            ent[(1 + V) * i] = ldg_stream_b32(a.colIdx + k, stream);
#pragma unroll
            for (int w = 0; w < V; ++w)
                ent[(1 + V) * i + 1 + w] = ldg_stream_b32(a.val + (int64_t)k * V + w, stream);
        }
    }
}

// What a launch hands its kernel: no more than the kernel reads (SpmmLongArgs).
template <bool LONG, bool RAGGED>
using SpmmKernelArgs = std::conditional_t<RAGGED, SpmmRaggedArgs, std::conditional_t<LONG, SpmmLongArgs, SpmmArgs>>;

// Words of shared memory per lane group.  A RAGGED row passes through a row of them on its way out, so that the lanes store
// neighbouring floats: the four of a lane one by one are four times the sectors (3.2 M entries at 47 columns, split: 96 us,
// this way 85; shifted to whole 16-byte vectors with single floats at the ends 92: bank conflicts and divergence).
template <int LPR, int VW, int CF, int V, bool RAGGED>
constexpr int spmm_group_words = SpmmTile<LPR, V>::GROUP_WORDS + (RAGGED ? LPR * CF * VW : 0);

// MLP = 16-byte gathers a lane keeps in flight per batch (2, 4, 8 or 16).  It trades registers
// (and so resident warps per SM) against memory-level parallelism inside one warp; the
// launch bound asks for the matching number of resident 256-thread CTAs.
template <int MLP>
struct SpmmOcc {
    static constexpr int MIN_CTAS = MLP >= 16 ? 2 : (MLP >= 8 ? 3 : (MLP >= 4 ? 5 : 8));
};

// ACC = true adds the product to C instead of overwriting it: every contribution is a RED, rows
// without entries add nothing, and nothing is zeroed (no pre-pass either).
// LONG = true (unsplit layouts) passes over rows of more than PSPMM_LONG_ROW entries
// (long_rows.cuh); its first CTAs prepare the launch that takes them.  Both are template
// flags because a run-time test of either costs the 48- and 80-register shapes spills (4 - 13 % of
// the dim sweep's products).
// RAGGED = true: see SpmmRaggedArgs.  Only what is stored differs.
template <int LPR, int VW, int CF, int V, int MLP, bool ACC = false, bool LONG = false, bool RAGGED = false>
__global__ void __launch_bounds__(256, SpmmOcc<MLP>::MIN_CTAS) spmm_seg_kernel(const SpmmKernelArgs<LONG, RAGGED> a)
{
    using Tile = SpmmTile<LPR, V>;
    constexpr int CAP = Tile::CAP;
    constexpr int U0 = MLP / (CF * (V > 1 ? 2 : 1));
    // entries per full gather batch: a power of two (the row tail falls through U/2, U/4, ...)
    constexpr int U = U0 >= 16 ? 16 : (U0 >= 8 ? 8 : (U0 >= 4 ? 4 : (U0 >= 2 ? 2 : 1)));

    extern __shared__ __align__(16) int smem_words[];
    const int gpc = blockDim.x / LPR;
    const int g = threadIdx.x / LPR;
    const int gl = threadIdx.x % LPR;
    const unsigned gmask =
        (LPR == 32) ? PSPMM_FULL_MASK : (((1u << LPR) - 1u) << (((threadIdx.x & 31) / LPR) * LPR));
    int *sp = smem_words + g * spmm_group_words<LPR, VW, CF, V, RAGGED>;  // segment pointers
    int *st = sp + (PSPMM_RPG_MAX + 1);                     // target rows: [0] previous, [1..] own, then next
    int *ent = sp + Tile::HEAD_WORDS;                       // staged entries

    const int rpg = a.rows_per_group;
    int64_t first = ((int64_t)blockIdx.x * gpc + g) * rpg;
    if constexpr (LONG) {
        pdl_launch_dependents();
        if (blockIdx.x < (unsigned)a.lng.scan_ctas) {
            if (blockIdx.y == 0)
                long_scan(a.lng, a.segPtr, a.n_seg, (int)blockIdx.x);
            return;
        }
        first -= (int64_t)a.lng.scan_ctas * gpc * rpg;
    }
    if (first >= a.n_seg)
        return;  // the whole group leaves; groups only ever synchronise among themselves
    const int nrow = (a.n_seg - first < rpg) ? (int)(a.n_seg - first) : rpg;
    const bool split = a.target_row != nullptr;

    for (int i = gl; i <= nrow; i += LPR)
        sp[i] = __ldg(a.segPtr + first + i);
    if (split) {
        for (int i = gl; i < nrow + 2; i += LPR) {
            const int64_t s = first - 1 + i;
            st[i] = (s < 0) ? -1 : (s >= a.n_seg ? (int)a.n_out : __ldg(a.target_row + s));
        }
    }

    // Per-lane column slices; lanes past the last column read slice 0 and never store.
    const int vec0 = blockIdx.y * (LPR * CF);
    bool act[CF];
    int voff[CF];
    const char *bcol[CF];
#pragma unroll
    for (int cf = 0; cf < CF; ++cf) {
        const int v = vec0 + cf * LPR + gl;
        act[cf] = v < a.nvec;
        voff[cf] = act[cf] ? v * VW : 0;
        bcol[cf] = reinterpret_cast<const char *>(a.B + voff[cf]);
    }
    const unsigned ldB_bytes = (unsigned)(a.ldB * 4);
    // B is gathered many times: keep a stable fraction of it in L2.  A is read once and C is
    // written once: both are marked evict-first so they do not push B out.
    const unsigned long long keep = l2_policy_keep(a.keep_fraction);
    const unsigned long long stream = l2_policy_stream();

    float acc[V][CF][VW];
#pragma unroll
    for (int w = 0; w < V; ++w)
#pragma unroll
        for (int cf = 0; cf < CF; ++cf)
#pragma unroll
            for (int i = 0; i < VW; ++i)
                acc[w][cf][i] = 0.f;

    if (split)
        pdl_wait();  // the pre-pass has zeroed the rows that are added to
    __syncwarp(gmask);
    int cur = sp[0];
    const int end = sp[nrow];
    int row = 0;
    int run_start = 0;  // first of the group's segments accumulated into the current row
    bool head_pending = (first == 0);  // the rows ahead of the very first segment are still to be zeroed
    while (true) {
        const int fill = (end - cur < CAP) ? (end - cur) : CAP;
        spmm_stage<LPR, V>(a, ent, cur, fill, gl, stream);
        __syncwarp(gmask);
        const int lim = cur + fill;
        int resume = lim;
        while (row < nrow) {
            const int rb = sp[row], re = sp[row + 1];
            const bool skip = LONG && re - rb > PSPMM_LONG_ROW;  // left to spmm_long_rows_kernel
            const int e = (rb > cur ? rb : cur) - cur;
            const int eh = skip ? e : (re < lim ? re : lim) - cur;
            spmm_entries<U, LPR, VW, CF, V>(ent, e, eh, bcol, ldB_bytes, keep, acc);
            if (re > lim && !skip)
                break;  // the row continues in the next window

            // ---- the segment is complete
            int64_t orow = first + row;
            bool shared = false;
            int next = 0;
            if (split && a.bucketed) {
                // Length-bucketed plan: segments in any order, flags in the high bits of the target.
                const unsigned me = (unsigned)st[row + 1];
                const unsigned nx = (unsigned)st[row + 2];
                if (row + 1 < nrow && ((nx ^ me) & PSPMM_SEG_ROW_MASK) == 0) {
                    ++row;  // the group's next segment is another piece of the same row
                    continue;
                }
                orow = me & PSPMM_SEG_ROW_MASK;
                shared = (me & PSPMM_SEG_MULTI) != 0;
            } else if (split) {
                const int me = st[row + 1];
                next = st[row + 2];
                if (next == me && row + 1 < nrow) {
                    ++row;  // the group's next segment continues the same row: keep accumulating
                    continue;
                }
                orow = me;
                // Pieces of this row held by other groups add into it as well.
                shared = (run_start == 0 && st[0] == me) || (next == me);
                run_start = row + 1;
            }
            // (pieces of a split layout are never empty)
            const bool emit = (!ACC || split || re > rb) && !skip;
#pragma unroll
            for (int w = 0; w < V; ++w) {
                float *crow = a.C + (orow * V + w) * a.ldC;
#pragma unroll
                for (int cf = 0; cf < CF; ++cf) {
                    if constexpr (RAGGED) {
                        st_vec<VW>(reinterpret_cast<float *>(ent + CAP * (1 + V)) + (cf * LPR + gl) * VW, acc[w][cf]);
                    } else if (act[cf] && emit) {
                        if (ACC || shared)
                            red_add_vec<VW>(crow + voff[cf], acc[w][cf]);
                        else
                            st_vec_hint<VW>(crow + voff[cf], acc[w][cf], stream);
                    }
#pragma unroll
                    for (int i = 0; i < VW; ++i)
                        acc[w][cf][i] = 0.f;
                }
                if constexpr (RAGGED) {
                    const float *out = reinterpret_cast<float *>(ent + CAP * (1 + V));
                    const int left = a.dim - vec0 * VW, cols = left < LPR * CF * VW ? left : LPR * CF * VW;
                    float *to = crow + vec0 * VW;
                    __syncwarp(gmask);
                    for (int j = emit ? gl : cols; j < cols; j += LPR) {
                        if (shared)
                            red_add_vec<1>(to + j, out + j);
                        else
                            st_vec_hint<1>(to + j, out + j, stream);
                    }
                    __syncwarp(gmask);
                }
            }
            if (!ACC && split && !a.bucketed) {
                // Rows strictly between this segment's row and the next segment's row (and, for
                // the very first segment, the rows before it) have no entries: zero short runs
                // here; runs longer than PSPMM_GAP_MAX are left to the pre-pass.
                const float zero[VW] = {};
                auto zero_rows = [&](int64_t r0, int64_t r1) {
                    for (int64_t r = r0 * V; r < r1 * V; ++r) {
                        float *crow = a.C + r * a.ldC;
#pragma unroll
                        for (int cf = 0; cf < CF; ++cf)
                            if (act[cf]) {
                                if constexpr (RAGGED)
                                    for (int i = 0; i < VW && voff[cf] + i < a.dim; ++i)
                                        st_vec_hint<1>(crow + voff[cf] + i, zero, stream);
                                else
                                    st_vec_hint<VW>(crow + voff[cf], zero, stream);
                            }
                    }
                };
                const int64_t after = (int64_t)next - orow - 1;
                if (after > 0 && after <= PSPMM_GAP_MAX)
                    zero_rows(orow + 1, next);
                if (head_pending && orow > 0 && orow <= PSPMM_GAP_MAX)
                    zero_rows(0, orow);
                head_pending = false;
            }
            ++row;
            if (skip) {  // the window restarts behind the long row
                resume = re;
                break;
            }
        }
        if (row >= nrow)
            break;
        cur = resume;
        __syncwarp(gmask);  // everyone is done reading the window before it is refilled
    }
}

// The long rows of an unsplit (block-)CSR layout (long_rows.cuh), which spmm_seg_kernel passes over.
// The entries of a share are dealt to the lane groups in equal spans, which they walk as
// spmm_seg_kernel walks its segments.  Every sum has a fixed order, as without the cut: the pieces of a
// row inside a share meet in shared memory in the order of the entries, the shares' parts in
// a.lng.partials.  Bound: gather latency (U loads of 16 bytes in flight per lane).
template <int VW, int V, int LPR, bool RAGGED = false>
__global__ void __launch_bounds__(256, 3) spmm_long_rows_kernel(const SpmmKernelArgs<true, RAGGED> a)
{
    constexpr int G = 256 / LPR;
    constexpr int U = V > 1 ? 4 : 8;
    constexpr int CAP = SpmmTile<LPR, V>::CAP;
    constexpr int ROW = LPR * VW;  // columns of this CTA
    constexpr int WINDOW_WORDS = G * CAP * (1 + V), PART_WORDS = G * 2 * V * ROW;
    __shared__ __align__(16) int work[WINDOW_WORDS > PART_WORDS ? WINDOW_WORDS : PART_WORDS];  // windows, then parts
    __shared__ LongShare::Shared sh;
    float *parts = reinterpret_cast<float *>(work);
    const int lane = threadIdx.x & 31;
    const int g = threadIdx.x / LPR, gl = lane % LPR;
    const unsigned gmask = (LPR == 32) ? PSPMM_FULL_MASK : (((1u << LPR) - 1u) << ((lane / LPR) * LPR));
    int *ent = work + g * CAP * (1 + V);
    const int v = blockIdx.y * LPR + gl;
    const bool act = v < a.nvec;
    const int voff = act ? v * VW : 0;
    const char *bcol[1] = {reinterpret_cast<const char *>(a.B + voff)};
    const unsigned ldB_bytes = (unsigned)(a.ldB * 4);
    const unsigned long long keep = l2_policy_keep(a.keep_fraction);
    const unsigned long long stream = l2_policy_stream();
    const int64_t dimv = (int64_t)a.nvec * VW;  // columns of a partial result
    int64_t dim = dimv;
    if constexpr (RAGGED)
        dim = a.dim;
    const int share = blockIdx.x;
    float acc[V][1][VW], first[V][VW];

    // Few rows: the CTAs find their shares without the segment kernel and gather beside it; only the counters, which it
    // clears, are waited for.  (It writes none of these rows.  19.7 K rows, 197 K entries, dim 16: the two took 9.5 and 8 us
    // one behind the other.)  Every CTA waits for it once, so that this launch does not end before it.
    __shared__ int own[PSPMM_OWN_TOTALS];
    if (a.lng.own_totals) {
        long_own_totals(own, a.lng, a.segPtr, a.n_seg);
        __syncthreads();
    } else {
        pdl_wait();
    }
    LongShare job;
    if (!job.begin(a.lng, sh, share, a.lng.own_totals ? own : nullptr)) {
        pdl_wait();
        return;
    }
    while (job.look(sh, a.segPtr, a.n_seg)) {
        const int total = job.total;
        if (total == 0)
            continue;
        // What a row sums up to in this share: the result, or its part of it.
        auto emit = [&](int i, int w, int col, const float *val) {
            int s0, s1;
            job.shares_of(sh, i, s0, s1);
            float *to = a.C + ((int64_t)sh.row[i] * V + w) * a.ldC + col;
            if constexpr (RAGGED) {
                if (s0 == s1) {
#pragma unroll
                    for (int j = 0; j < VW; ++j)
                        if (col + j < dim)
                            st_vec_hint<1>(to + j, val + j, stream);
                    return;
                }
            }
            if (s0 == s1)
                st_vec_hint<VW>(to, val, stream);
            else
                st_vec<VW>(a.lng.partials + (LongShare::slot(share, s0) * V + w) * dimv + col, val);
        };
        const int span = ((total + G - 1) / G + U - 1) / U * U;
        const int start = g * span;
        const int stop = start + span < total ? start + span : total;
        int p = start;  // position in the concatenation
        int i = p < stop ? job.row_of(sh, p) : 0;
        bool has_first = false, has_last = false;
        while (p < stop) {
            const bool from_row_start = p == job.off(sh, i), from_span_start = p == start;
            const int row_end = job.off(sh, i + 1), row_stop = row_end < stop ? row_end : stop;
            const int from = sh.lo[i] - job.off(sh, i);
#pragma unroll
            for (int w = 0; w < V; ++w)
#pragma unroll
                for (int j = 0; j < VW; ++j)
                    acc[w][0][j] = 0.f;
            while (p < row_stop) {
                const int fill = row_stop - p < CAP ? row_stop - p : CAP;
                spmm_stage<LPR, V>(a, ent, from + p, fill, gl, stream);
                __syncwarp(gmask);
                spmm_entries<U, LPR, VW, 1, V, true>(ent, 0, fill, bcol, ldB_bytes, keep, acc);
                __syncwarp(gmask);
                p += fill;
            }
            if (from_row_start && p == row_end) {  // all of the row's entries in this share
                if (act) {
#pragma unroll
                    for (int w = 0; w < V; ++w)
                        emit(i, w, voff, acc[w][0]);
                }
                has_last = false;
            } else if (from_span_start) {
                has_first = true;
#pragma unroll
                for (int w = 0; w < V; ++w)
#pragma unroll
                    for (int j = 0; j < VW; ++j)
                        first[w][j] = acc[w][0][j];
            } else {
                has_last = true;  // (only the span's last piece ends inside a row)
            }
            ++i;
        }
        __syncthreads();  // the windows are free
#pragma unroll
        for (int w = 0; w < V; ++w)
#pragma unroll
            for (int j = 0; j < VW; ++j) {
                if (has_first)
                    parts[((g * 2) * V + w) * ROW + gl * VW + j] = first[w][j];
                if (has_last)
                    parts[((g * 2 + 1) * V + w) * ROW + gl * VW + j] = acc[w][0][j];
            }
        __syncthreads();
        // Rows that several groups share, their pieces in order.
        const int row0 = sh.edge[0], rows = sh.edge[1] - row0 + 1;
        for (int t = threadIdx.x; t < rows * V * LPR; t += 256) {
            const int i2 = row0 + t / (V * LPR), w = t / LPR % V, l = t % LPR;
            const int vi = blockIdx.y * LPR + l;
            const int off0 = job.off(sh, i2);
            const int g0 = off0 / span, g1 = (job.off(sh, i2 + 1) - 1) / span;
            if (g0 == g1 || vi >= a.nvec)
                continue;  // one group had all of it
            float sum[VW];
#pragma unroll
            for (int j = 0; j < VW; ++j)
                sum[j] = 0.f;
            for (int q = g0; q <= g1; ++q) {
                const int slot = q > g0 || off0 == q * span ? 0 : 1;
#pragma unroll
                for (int j = 0; j < VW; ++j)
                    sum[j] += parts[((q * 2 + slot) * V + w) * ROW + l * VW + j];
            }
            emit(i2, w, vi * VW, sum);
        }
        pdl_wait();  // (the counters; no wait but the first)
        job.arrive(a.lng, sh, blockIdx.y, gridDim.y);
        for (int q = 0; q < 2; ++q) {
            if (!sh.last[q])
                continue;
            int s0, s1;
            job.shares_of(sh, sh.edge[q], s0, s1);
            const int64_t r = sh.row[sh.edge[q]];
            for (int t = threadIdx.x; t < V * ROW; t += 256) {
                const int w = t / ROW, col = blockIdx.y * ROW + t % ROW;
                if (col >= dim)
                    continue;
                float sum = 0.f;
                for (int c = s0; c <= s1; ++c)
                    sum += __ldcg(a.lng.partials + (LongShare::slot(c, s0) * V + w) * dimv + col);
                a.C[(r * V + w) * a.ldC + col] = sum;
            }
        }
        __syncthreads();
    }
    pdl_wait();
}

template <int VW, int V, bool RAGGED = false>
static inline void spmm_launch_long_rows(const SpmmKernelArgs<true, RAGGED> &a, cudaStream_t st)
{
    const int lpr = pspmm_long_lanes(a.nvec, V);
    const dim3 grid((unsigned)a.lng.shares, (unsigned)((a.nvec + lpr - 1) / lpr));
    if (lpr == 32)
        launch_dependent(spmm_long_rows_kernel<VW, V, 32, RAGGED>, grid, 256, 0, st, a);
    else if (lpr == 16)
        launch_dependent(spmm_long_rows_kernel<VW, V, 16, RAGGED>, grid, 256, 0, st, a);
    else if constexpr (V == 1) {
        if (lpr == 8)
            launch_dependent(spmm_long_rows_kernel<VW, V, 8, RAGGED>, grid, 256, 0, st, a);
        else
            launch_dependent(spmm_long_rows_kernel<VW, V, 4, RAGGED>, grid, 256, 0, st, a);
    }
}

// The launch that follows spmm_seg_kernel when rows may have been left to it.
#define PSPMM_SPMM_LONG_ROWS(VW_)                                            \
    if (a.lng.totals) {                                                      \
        if (V == 1)                                                          \
            spmm_launch_long_rows<VW_, 1>(a, st);                            \
        else if (V == 2)                                                     \
            spmm_launch_long_rows<VW_, 2>(a, st);                            \
        else                                                                 \
            spmm_launch_long_rows<VW_, 3>(a, st);                            \
    }

template <int LPR, int VW, int CF, int V, int MLP, bool ACC = false, bool LONG = false, bool RAGGED = false>
static inline void spmm_launch_one(const SpmmKernelArgs<true, RAGGED> &a, dim3 grid, int threads, cudaStream_t st)
{
    const int smem = (threads / LPR) * spmm_group_words<LPR, VW, CF, V, RAGGED> * 4;
    auto kern = spmm_seg_kernel<LPR, VW, CF, V, MLP, ACC, LONG, RAGGED>;
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    const SpmmKernelArgs<LONG, RAGGED> &args = a;
    if (a.dependent)
        launch_dependent(kern, grid, threads, smem, st, args);  // follows the zeroing pre-pass
    else
        kern<<<grid, threads, smem, st>>>(args);
}

// Expands to the dispatch over the instantiated (LPR, CF) pairs of one (VW, V).
// (the form that passes over long rows is built at one gather-batch depth)
#define PSPMM_SPMM_CASE(LPR_, CF_, VW_, V_)                                               \
    if (s.lpr == LPR_ && s.cf == CF_) {                                                   \
        if (a.lng.totals)                                                       \
            spmm_launch_one<LPR_, VW_, CF_, V_, 8, false, true>(a, grid, s.threads, st);  \
        else                                                                              \
            spmm_launch_one<LPR_, VW_, CF_, V_, 8>(a, grid, s.threads, st);               \
        return true;                                                                      \
    }
// Same, with every gather-batch depth instantiated (used for the 128-bit CSR family).
#define PSPMM_SPMM_CASE_MLP(LPR_, CF_, VW_, V_)                              \
    if (s.lpr == LPR_ && s.cf == CF_) {                                      \
        if (a.lng.totals)                                          \
            spmm_launch_one<LPR_, VW_, CF_, V_, 8, false, true>(a, grid, s.threads, st); \
        else if (s.mlp == 2)                                                 \
            spmm_launch_one<LPR_, VW_, CF_, V_, 2>(a, grid, s.threads, st);  \
        else if (s.mlp == 4)                                                 \
            spmm_launch_one<LPR_, VW_, CF_, V_, 4>(a, grid, s.threads, st);  \
        else if (s.mlp == 16)                                                \
            spmm_launch_one<LPR_, VW_, CF_, V_, 16>(a, grid, s.threads, st); \
        else                                                                 \
            spmm_launch_one<LPR_, VW_, CF_, V_, 8>(a, grid, s.threads, st);  \
        return true;                                                         \
    }
#define PSPMM_SPMM_CASE_RAGGED(LPR_, CF_)                                                        \
    if (s.lpr == LPR_ && s.cf == CF_) {                                                          \
        if (a.lng.totals)                                                                        \
            spmm_launch_one<LPR_, 4, CF_, 1, 8, false, true, true>(a, grid, s.threads, st);      \
        else if (s.mlp <= 4)                                                                     \
            spmm_launch_one<LPR_, 4, CF_, 1, 4, false, false, true>(a, grid, s.threads, st);     \
        else if (s.mlp == 16)                                                                    \
            spmm_launch_one<LPR_, 4, CF_, 1, 16, false, false, true>(a, grid, s.threads, st);    \
        else                                                                                     \
            spmm_launch_one<LPR_, 4, CF_, 1, 8, false, false, true>(a, grid, s.threads, st);     \
        return true;                                                                             \
    }
// The accumulating form is built for the 128-bit CSR family at one gather-batch depth.
#define PSPMM_SPMM_CASE_ACC(LPR_, CF_)                                       \
    if (s.lpr == LPR_ && s.cf == CF_) {                                      \
        spmm_launch_one<LPR_, 4, CF_, 1, 8, true>(a, grid, s.threads, st);   \
        return true;                                                         \
    }
