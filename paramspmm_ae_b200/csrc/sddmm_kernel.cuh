// Segment SDDMM kernel for sm_100a: out[k] = <A[row(k)], B[colIdx[k]]> on a sparsity pattern.
//
// Same work decomposition as the SpMM kernel: a group of LPR lanes owns one segment (CSR
// row, PCSR row piece, or a V x 1 block-row form), lane gl holds the slice
// [(cf*LPR + gl)*VW, +VW), cf < CF, of the segment's A row(s) in registers and multiplies it
// with the same slice of every gathered B row (128-bit loads for VW = 4).
//
// The per-entry lane partials are not reduced one entry at a time.  LPR entries are
// processed together and reduced with a recursive-halving exchange: at stride s each lane
// keeps the half of the entries selected by its own lane bit and ships the other half to
// lane ^ s.  After log2(LPR) rounds lane gl owns the complete dot product of entry gl of
// the batch, at a cost of LPR-1 shuffles per LPR entries (about one per entry instead of
// log2(LPR)), and the results leave as one coalesced store per group.
#pragma once

#include "pspmm_common.cuh"
#include "vec_ops.cuh"

// p[0..N) per lane -> returns, on lane gl of each LPR-wide group, the sum over the group of p[gl].
template <int N>
__device__ __forceinline__ float transpose_reduce(float (&p)[N], int gl)
{
    if constexpr (N == 1) {
        return p[0];
    } else {
        constexpr int H = N / 2;
        float q[H];
        const bool upper = (gl & H) != 0;
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const float keep = upper ? p[i + H] : p[i];
            const float send = upper ? p[i] : p[i + H];
            q[i] = keep + __shfl_xor_sync(PSPMM_FULL_MASK, send, H);
        }
        return transpose_reduce<H>(q, gl);
    }
}

// The entries [lb, hb) of (block-)row arow for one lane group; every lane of the warp calls this
// together, `maxlen` is the longest of the warp's ranges and a group without work passes lb == hb.
template <int LPR, int VW, int CF, int V>
__device__ __forceinline__ void sddmm_entries(const SddmmArgs &a, int64_t arow, int lb, int hb, int maxlen, int gl)
{
    constexpr int ENT = (LPR >= 16) ? 1 : (16 / LPR);
    constexpr int CHUNK = LPR * ENT;
    // entries whose gathers are batched (divides LPR): 8 loads in flight per lane, 16 with wide rows
    constexpr int U0 = CF >= 8 ? 2 : (CF >= 3 ? 4 : 8 / CF);
    constexpr int U1 = V > 1 && U0 > 1 && CF > 1 ? U0 / 2 : U0;
    constexpr int U = U1 > LPR ? LPR : U1;
    const int tiles = (a.nvec + LPR * CF - 1) / (LPR * CF);
    const int len = hb - lb;
    const unsigned ub = lb, ue = hb;  // (lb and maxlen can add up to more than 2^31)
    const bool live = len > 0;
    const unsigned ldB_lo = (unsigned)(a.ldB * 4), ldB_hi = (unsigned)((unsigned long long)(a.ldB * 4) >> 32);
    // With several slices per lane a row that is not loaded keeps what was there, and what comes of it is not stored
    // (the scores of entries beyond the segment) or left out (slices beyond the last column).  Clearing it took an
    // instruction per float: 4 M entries, dim 100 170 -> 158 us, 256 378 -> 317; 0.9 M unsplit, dim 256 158 -> 109.  With one
    // slice the compiler overlaps batches if it may clear (band of 24 at dim 16: 60 us, without 75).
    constexpr bool KEEP = V == 1 && CF > 1 && (CF <= 4 || VW < 4);
    FVec<VW> kept[KEEP ? U : 1][KEEP ? CF : 1];
    if constexpr (KEEP) {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int cf = 0; cf < CF; ++cf)
                kept[u][cf] = zero_vec<VW>();
    }
    for (int off = 0; off < maxlen; off += CHUNK) {
        int ccol[ENT];
        float cval[ENT][V];
        float res[ENT][V];
#pragma unroll
        for (int t = 0; t < ENT; ++t) {
            const unsigned k = ub + off + t * LPR + gl;
            const bool ok = k < ue;
            ccol[t] = ok ? __ldg(a.colIdx + k) : 0;
#pragma unroll
            for (int w = 0; w < V; ++w) {
                cval[t][w] = (V > 1 && ok) ? __ldg(a.val + (int64_t)k * V + w) : 1.f;
                res[t][w] = 0.f;
            }
        }
        const int cnt = len - off;
        const int wcnt = maxlen - off;

        for (int tile = 0; tile < tiles; ++tile) {
            // Slice of the A row(s) this lane is responsible for in this tile.
            FVec<VW> av[V][CF];
            int voff[CF];
            bool act[CF];
#pragma unroll
            for (int cf = 0; cf < CF; ++cf) {
                const int vi = (tile * CF + cf) * LPR + gl;
                act[cf] = vi < a.nvec;
                voff[cf] = vi * VW;
#pragma unroll
                for (int w = 0; w < V; ++w)
                    // (the last block-row of an odd row count has lanes without a row of A)
                    av[w][cf] = (live && act[cf] && arow * V + w < a.n_rows_A)
                                    ? ldg_vec<VW>(a.A + (arow * V + w) * a.ldA + voff[cf])
                                    : zero_vec<VW>();
            }
#pragma unroll
            for (int t = 0; t < ENT; ++t) {
                if (t * LPR >= wcnt)
                    break;
                float part[V][LPR];
#pragma unroll
                for (int j0 = 0; j0 < LPR; j0 += U) {
                    FVec<VW> cleared[KEEP ? 1 : U][KEEP ? 1 : CF];
                    auto x = [&](int u, int cf) -> FVec<VW> & {
                        if constexpr (KEEP)
                            return kept[u][cf];
                        else
                            return cleared[u][cf];
                    };
                    const bool batch_on = (t * LPR + j0) < wcnt;  // warp-uniform
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int e = t * LPR + j0 + u;
                        const int c = __shfl_sync(PSPMM_FULL_MASK, ccol[t], j0 + u, LPR);
                        const bool p = batch_on && (e < cnt);
                        if constexpr (KEEP) {
                            const float *brow = row_start(a.B + voff[0], c, ldB_lo, ldB_hi);
#pragma unroll
                            for (int cf = 0; cf < CF; ++cf)
                                ldg_vec_keep<VW>(x(u, cf), brow + cf * LPR * VW, p && act[cf]);
                        } else {
                            const float *brow = a.B + (int64_t)c * a.ldB;
#pragma unroll
                            for (int cf = 0; cf < CF; ++cf)
                                x(u, cf) = ldg_vec_if<VW>(brow + voff[cf], p && act[cf]);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int w = 0; w < V; ++w) {
                            float s = 0.f;
#pragma unroll
                            for (int cf = 0; cf < CF; ++cf)
                                if (!KEEP || act[cf]) {
#pragma unroll
                                    for (int i = 0; i < VW; ++i)
                                        s = fmaf(av[w][cf].v[i], x(u, cf).v[i], s);
                                }
                            part[w][j0 + u] = s;
                        }
                }
#pragma unroll
                for (int w = 0; w < V; ++w)
                    res[t][w] += transpose_reduce<LPR>(part[w], gl);
            }
        }
#pragma unroll
        for (int t = 0; t < ENT; ++t) {
            const unsigned k = ub + off + t * LPR + gl;
            if (k < ue) {
#pragma unroll
                for (int w = 0; w < V; ++w) {
                    // Block layouts: positions whose stored value is zero are not part of
                    // the pattern and receive zero.
                    const float r = (V > 1 && cval[t][w] == 0.f) ? 0.f : res[t][w];
                    __stcs(a.out + (int64_t)k * V + w, r);
                }
            }
        }
    }
}

// The first `long_ctas` CTAs look after the long rows (more than a.long_row entries), which the lane
// groups of the others pass over: a hub row is otherwise one group's serial walk (25 K entries, dim
// 100: 8.8 ms in a product whose other rows take 0.1 ms).  CTA c owns the entries
// [c, c+1) * a.long_range, finds the long rows among them (find_segment, then one look at each row
// between) and deals pieces of their entries to its lane groups.  Entries are independent, so nothing
// has to be merged and one launch does both.
template <int LPR, int VW, int CF, int V>
__global__ void __launch_bounds__(512) sddmm_seg_kernel(const SddmmArgs a)
{
    const int gpc = blockDim.x / LPR;
    const int g = threadIdx.x / LPR;
    const int gl = threadIdx.x % LPR;

    if (blockIdx.x < a.long_ctas) {
        __shared__ int row_list[PSPMM_LONG_LIST], row_lo[PSPMM_LONG_LIST], row_hi[PSPMM_LONG_LIST];
        __shared__ int row_ends[2];
        __shared__ int n_long;
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int64_t begin = __ldg(a.segPtr), end = __ldg(a.segPtr + a.n_seg);
        for (int64_t s = begin + (int64_t)blockIdx.x * a.long_range; s < end; s += (int64_t)a.long_ctas * a.long_range) {
            const int64_t e1 = s + a.long_range < end ? s + a.long_range : end;
            if (threadIdx.x == 0)
                n_long = 0;
            for (int q = warp; q < 2; q += blockDim.x >> 5) {
                const int r = find_segment(a.segPtr, a.n_seg, begin, end, q == 0 ? s : e1 - 1, lane);
                if (lane == 0)
                    row_ends[q] = r;
            }
            __syncthreads();
            for (int64_t r = row_ends[0] + threadIdx.x; r <= row_ends[1]; r += blockDim.x) {
                const int64_t rb = __ldg(a.segPtr + r), re = __ldg(a.segPtr + r + 1);
                if (re - rb > a.long_row) {
                    const int i = atomicAdd(&n_long, 1);
                    row_list[i] = (int)r;
                    row_lo[i] = (int)(rb > s ? rb : s);
                    row_hi[i] = (int)(re < e1 ? re : e1);
                }
            }
            __syncthreads();
            // Pieces of 32 entries, dealt to the lane groups in turn over all long rows of the range.  (16 for narrow groups of
            // several slices: they are more to a CTA, and each takes longer.)
            constexpr int PIECE = LPR <= 8 && CF > 1 && V == 1 ? 16 : 32;
            const int n = n_long;
            int i = 0, piece0 = 0;  // the row the group stands in, and the number of its first piece
            for (int p0 = 0;; p0 += gpc) {
                const int p = p0 + g;
                int pieces = 0;
                while (i < n && p >= piece0 + (pieces = (row_hi[i] - row_lo[i] + PIECE - 1) / PIECE)) {
                    piece0 += pieces;
                    ++i;
                }
                if (!__any_sync(PSPMM_FULL_MASK, i < n))
                    break;  // (pieces are dealt in order: the warp has none left)
                int lb = 0, hb = 0;
                int64_t row = 0;
                if (i < n) {
                    row = row_list[i];
                    lb = row_lo[i] + (p - piece0) * PIECE;
                    hb = row_hi[i] - lb > PIECE ? lb + PIECE : row_hi[i];
                }
                sddmm_entries<LPR, VW, CF, V>(a, row, lb, hb, PIECE, gl);
            }
            __syncthreads();
        }
        return;
    }

    const int64_t seg0 = (int64_t)(blockIdx.x - a.long_ctas) * gpc * a.rows_per_group;
    for (int it = 0; it < a.rows_per_group; ++it) {
        const int64_t seg = seg0 + (int64_t)it * gpc + g;
        int lb = 0, hb = 0;
        int64_t arow = 0;
        if (seg < a.n_seg) {
            lb = __ldg(a.segPtr + seg);
            hb = __ldg(a.segPtr + seg + 1);
            arow = a.target_row ? (int64_t)__ldg(a.target_row + seg) : seg;
            if (hb - lb > a.long_row)
                hb = lb;
        }
        int maxlen = hb - lb;
        if constexpr (LPR < 32)
            maxlen = __reduce_max_sync(PSPMM_FULL_MASK, maxlen);
        sddmm_entries<LPR, VW, CF, V>(a, arow, lb, hb, maxlen, gl);
    }
}

template <int LPR, int VW, int CF, int V>
static inline void sddmm_launch_one(const SddmmArgs &a, dim3 grid, int threads, cudaStream_t st)
{
    sddmm_seg_kernel<LPR, VW, CF, V><<<grid, threads, 0, st>>>(a);
}

#define PSPMM_SDDMM_CASE(LPR_, CF_, VW_, V_)                             \
    if (s.lpr == LPR_ && s.cf == CF_) {                                  \
        sddmm_launch_one<LPR_, VW_, CF_, V_>(a, grid, s.threads, st);    \
        return true;                                                     \
    }
