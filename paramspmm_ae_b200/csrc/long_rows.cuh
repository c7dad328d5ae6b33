// Long rows of an unsplit layout: how their entries are dealt over the GPU.
//
// A kernel that gives every row to one lane group walks a long row's gather batches one after the
// other: a hub row of 1,600 entries held a 197 K-entry product at dim 16 for 310 us (98 % of it), and
// rows of a few hundred entries still leave the groups of a warp out of step.  Rows of more than
// PSPMM_LONG_ROW entries are therefore left to a second kernel, launched behind the first, whose CTAs
// take equal shares of all long rows' entries laid end to end.  Two steps prepare that, without any
// list in memory:
//   - the first CTAs of the first kernel (long_scan) add up the long rows' entries per 512 rows;
//   - a CTA of the second kernel (LongShare) finds its share in the running sum of those totals and
//     then looks at 512 rows at a time.
// (Shares by entry range of the whole matrix, found by binary search, left two thirds of the SMs idle
// on graphs whose hubs have neighbouring ids and cost the search per range: 62 us instead of 41 for
// 1.3 M entries in long rows at dim 16.)
//
// A row that ends up in several shares leaves one partial result per share; the share that brings the
// last one, by a counter that the first kernel clears, puts them together in order.
#pragma once

#include "pspmm_common.cuh"

// The first kernel's CTA `block` of scan_ctas (256 threads or fewer, whole warps): totals of 8 x 512 rows,
// and its part of the counters.
__device__ __forceinline__ void long_scan(const LongArgs &a, const int32_t *segPtr, int64_t n_seg, int block)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int64_t i = (int64_t)block * blockDim.x + threadIdx.x; i < a.n_counters; i += (int64_t)a.scan_ctas * blockDim.x)
        a.counters[i] = 0;
    for (int t = warp; t < 8; t += blockDim.x >> 5) {
        const int64_t r0 = ((int64_t)block * 8 + t) * PSPMM_LONG_ROWS;
        if (r0 >= n_seg)
            return;
        int sum = 0;
#pragma unroll 4
        for (int i = 0; i < PSPMM_LONG_ROWS / 32; ++i) {
            const int64_t r = r0 + i * 32 + lane;
            if (r < n_seg) {
                const int len = __ldg(segPtr + r + 1) - __ldg(segPtr + r);
                sum += len > PSPMM_LONG_ROW ? len : 0;
            }
        }
        sum = __reduce_add_sync(PSPMM_FULL_MASK, sum);
        if (lane == 0)
            a.totals[block * 8 + t] = sum;
    }
}

// The same totals, all of them, by one CTA of 256 threads for itself; segPtr lies on a 16-byte boundary.  One barrier is
// needed before they are read.  Bound: the latency of a warp's loads, so four pointers per load and the loads of two totals
// in flight, and the instructions of an SM's CTAs, so one or two per SM.  (One pointer per load and three CTAs: 20 K rows of 10, none
// long, 16 to 64 columns, 3.2 - 4.1 us longer than without this look, 32 K 5.2 - 6.2; now 2.0 - 2.3 and, at three CTAs, 4.  Clusters of four
// that share the look: 2 - 4, their launch alone 2.  The loads of four totals in flight spill.)
__device__ __forceinline__ void long_own_totals(int *totals, const LongArgs &a, const int32_t *segPtr, int64_t n_seg)
{
    constexpr int STEPS = PSPMM_LONG_ROWS / 128, TWO = 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int t0 = warp; t0 < a.n_totals; t0 += 8 * TWO) {
        int4 q[TWO][STEPS];
        int after[TWO];
#pragma unroll
        for (int u = 0; u < TWO; ++u) {
            const int r0 = (t0 + 8 * u) * PSPMM_LONG_ROWS;
            if (r0 + PSPMM_LONG_ROWS <= n_seg) {
#pragma unroll
                for (int i = 0; i < STEPS; ++i)
                    q[u][i] = __ldg(reinterpret_cast<const int4 *>(segPtr + r0) + i * 32 + lane);
                after[u] = __ldg(segPtr + r0 + PSPMM_LONG_ROWS);
            }
        }
#pragma unroll
        for (int u = 0; u < TWO; ++u) {
            const int t = t0 + 8 * u, r0 = t * PSPMM_LONG_ROWS;
            if (t >= a.n_totals)
                break;
            int sum = 0;
            if (r0 + PSPMM_LONG_ROWS <= n_seg) {
#pragma unroll
                for (int i = STEPS - 1; i >= 0; --i) {
                    const int4 x = q[u][i];
                    const int next = __shfl_down_sync(PSPMM_FULL_MASK, x.x, 1);
                    const int len[4] = {x.y - x.x, x.z - x.y, x.w - x.z, (lane < 31 ? next : after[u]) - x.w};
                    after[u] = __shfl_sync(PSPMM_FULL_MASK, x.x, 0);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        sum += len[j] > PSPMM_LONG_ROW ? len[j] : 0;
                }
            } else {  // the last rows
                for (int r = r0 + lane; r < n_seg; r += 32) {
                    const int len = __ldg(segPtr + r + 1) - __ldg(segPtr + r);
                    sum += len > PSPMM_LONG_ROW ? len : 0;
                }
            }
            sum = __reduce_add_sync(PSPMM_FULL_MASK, sum);
            if (lane == 0)
                totals[t] = sum;
        }
    }
}

// Inclusive sum over the 256 threads of a CTA; `warps` is scratch for 8 words.  One barrier before the
// result, and one is needed before the next use of `warps`.
template <typename T>
__device__ __forceinline__ T cta_scan(T x, T *warps, T *total)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T o = __shfl_up_sync(PSPMM_FULL_MASK, x, d);
        if (lane >= d)
            x += o;
    }
    if (lane == 31)
        warps[warp] = x;
    __syncthreads();
    T all = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        x += w < warp ? warps[w] : 0;
        all += warps[w];
    }
    *total = all;
    return x;
}

// What a share has to do, 512 rows at a time.  All 256 threads of the CTA call the members together.
//
// Positions ("units") run over the long rows' entries of the whole matrix, with PSPMM_LONG_LOOK units ahead
// of every 512 rows for the look at them, so that a share of few long rows among many short ones is no
// longer than the others.  They run to the entries plus one per row, beyond 2^31 for matrices near the index
// limit, and are 64 bits wide; what belongs to one share is not (long_fits).  Only look() knows positions: the
// users see offsets into the share's part of the look, and the 64-bit values stay out of their registers.
struct LongShare {
    struct Shared {
        int row[PSPMM_LONG_ROWS], lo[PSPMM_LONG_ROWS];  // the long rows of this look; their first entry in the share
        int off[PSPMM_LONG_ROWS + 1];                   // where they begin among its entries of the share
        unsigned long long warps[8];
        int64_t u0, u1, per;  // the share
        int64_t found[2];
        int edge[2];     // the rows that hold the first and the last entry of this look's part of the share
        int shares[2];   // the first share of the one, the last of the other
        int last[2];
    };
    int64_t pos;  // position of row r
    int64_t r;
    int share, total;  // total: entries of this look that belong to the share

    // False: nothing to do (no row is long, or fewer shares are needed than there are).  `own`: totals of
    // long_own_totals in shared memory, or nullptr.
    __device__ __forceinline__ bool begin(const LongArgs &a, Shared &sh, int share_, const int *own = nullptr)
    {
        const int tid = threadIdx.x;
        const int each = (a.n_totals + 255) / 256;
        unsigned long long mine = 0, all;
        bool any = false;
        share = share_;
#pragma unroll 8
        for (int i = 0; i < each; ++i) {
            const int t = tid * each + i;
            const int x = t >= a.n_totals ? 0 : (own ? own[t] : __ldcg(a.totals + t));
            any |= x > 0;
            mine += (unsigned long long)x + (t < a.n_totals ? PSPMM_LONG_LOOK : 0);
        }
        if (!__syncthreads_or(any))
            return false;
        const unsigned long long upto = cta_scan(mine, sh.warps, &all);
        const unsigned long long per = long_share_size((int64_t)all, a.shares);
        const unsigned long long first = share * per;
        if (first >= all)
            return false;
        if (tid == 0) {
            sh.u0 = (int64_t)first;
            sh.u1 = (int64_t)(all - first < per ? all : first + per);
            sh.per = (int64_t)per;
        }
        if (first >= upto - mine && first < upto) {
            unsigned long long before = upto - mine;
            int t = tid * each;
            while (true) {
                const unsigned long long x = (unsigned long long)(own ? own[t] : __ldcg(a.totals + t)) + PSPMM_LONG_LOOK;
                if (before + x > first)
                    break;
                before += x;
                ++t;
            }
            sh.found[0] = t;
            sh.found[1] = (int64_t)before;
        }
        __syncthreads();
        r = sh.found[0] * PSPMM_LONG_ROWS;
        pos = sh.found[1];
        return true;
    }

    // Looks at the next 512 rows.  False: the share ends.  total == 0: none of its entries lie here.
    __device__ __forceinline__ bool look(Shared &sh, const int32_t *segPtr, int64_t n_seg)
    {
        const int64_t u0 = sh.u0, u1 = sh.u1;
        if (pos >= u1)
            return false;
        int len[2], start[2];
        unsigned long long mine = 0, all;  // rows (high word) and entries
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int64_t q = r + 2 * threadIdx.x + i;
            start[i] = len[i] = 0;
            if (q < n_seg) {
                start[i] = __ldg(segPtr + q);
                len[i] = __ldg(segPtr + q + 1) - start[i];
                len[i] = len[i] > PSPMM_LONG_ROW ? len[i] : 0;
            }
            mine += (unsigned)len[i] + (len[i] ? 1ull << 32 : 0ull);
        }
        const unsigned long long before = cta_scan(mine, sh.warps, &all) - mine;
        const int64_t begin_at = pos + PSPMM_LONG_LOOK, end_at = begin_at + (unsigned)all;
        const int64_t base = u0 > begin_at ? u0 : begin_at;
        const int64_t part = (u1 < end_at ? u1 : end_at) - base;
        total = part > 0 ? (int)part : 0;
        int idx = (int)(before >> 32);
        int64_t at = begin_at + (unsigned)before - base;  // from the share's first entry of this look
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (len[i]) {
                const int64_t end = at + len[i];
                sh.row[idx] = (int)(r + 2 * threadIdx.x + i);
                sh.lo[idx] = start[i] + (at < 0 && end > 0 ? (int)-at : 0);
                sh.off[idx] = at < 0 ? 0 : (at < total ? (int)at : total);
                if (total) {
                    if (at <= 0 && end > 0) {
                        sh.edge[0] = idx;
                        sh.shares[0] = at == 0 ? share : (int)((base + at) / sh.per);
                    }
                    if (at < total && end >= total) {
                        sh.edge[1] = idx;
                        sh.shares[1] = end == total ? share : (int)((base + end - 1) / sh.per);
                    }
                }
                ++idx;
                at = end;
            }
        if (threadIdx.x == 0)
            sh.off[(int)(all >> 32)] = total;
        r += PSPMM_LONG_ROWS;
        pos = end_at;
        __syncthreads();
        return true;
    }

    // Where row i begins in the concatenation of this look's entries (the number of rows: where they end).
    __device__ __forceinline__ int off(const Shared &sh, int i) const { return sh.off[i]; }
    // The row that holds entry p of the concatenation.
    __device__ __forceinline__ int row_of(const Shared &sh, int p) const
    {
        int lo = sh.edge[0], hi = sh.edge[1] + 1;
        while (hi - lo > 1) {
            const int mid = (lo + hi) / 2;
            if (sh.off[mid] <= p)
                lo = mid;
            else
                hi = mid;
        }
        return lo;
    }
    // First and last share that row i is part of (edge[0] <= i <= edge[1]): only the outermost rows leave this one.
    __device__ __forceinline__ void shares_of(const Shared &sh, int i, int &s0, int &s1) const
    {
        s0 = i == sh.edge[0] ? sh.shares[0] : share;
        s1 = i == sh.edge[1] ? sh.shares[1] : share;
    }
    // Where a share's part of a row goes: slot 2 * share (the row began in an earlier share) or 2 * share + 1.
    __device__ __forceinline__ static int64_t slot(int share, int s0) { return 2 * (int64_t)share + (s0 == share ? 1 : 0); }

    // After the results of this look are stored: row sh.edge[q] (q = 0, 1) has sh.last[q] set if several
    // shares hold it and this CTA brought the last part.
    __device__ __forceinline__ void arrive(const LongArgs &a, Shared &sh, int tile, int tiles)
    {
        int s[4];
        shares_of(sh, sh.edge[0], s[0], s[1]);
        shares_of(sh, sh.edge[1], s[2], s[3]);
        const bool two = sh.edge[0] != sh.edge[1] && s[2] != s[3];
        if (s[0] == s[1] && !two) {
            __syncthreads();
            if (threadIdx.x < 2)
                sh.last[threadIdx.x] = 0;
            __syncthreads();
            return;
        }
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0)
            sh.last[0] = s[0] != s[1] && atomicAdd(a.counters + s[0] * tiles + tile, 1) == s[1] - s[0];
        if (threadIdx.x == 1)
            sh.last[1] = two && atomicAdd(a.counters + s[2] * tiles + tile, 1) == s[3] - s[2];
        __syncthreads();
        __threadfence();
    }
};
