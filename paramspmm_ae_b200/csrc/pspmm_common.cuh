// Shared declarations for the sm_100a kernels behind libpspmm's C ABI.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "pspmm.h"

#define PSPMM_FULL_MASK 0xffffffffu
#define PSPMM_MAX_CF 8
#define PSPMM_RPG_MAX 16  // most consecutive segments one lane group owns
#define PSPMM_LONG_RANGE_MAX 8192
#define PSPMM_LONG_LIST 132  // long rows that such a range can meet (8192 / 65 inside it and two cut), and a few
#define PSPMM_GAP_MAX 256  // longest run of uncovered rows the SpMM kernel zeroes by itself

// Records the CUDA error text for pspmm_last_cuda_error() and returns PSPMM_E_CUDA.
int pspmm_note_cuda_error(cudaError_t e);

#define PSPMM_CUDA_TRY(expr)                    \
    do {                                        \
        cudaError_t e__ = (expr);               \
        if (e__ != cudaSuccess)                 \
            return pspmm_note_cuda_error(e__);  \
    } while (0)

// Programmatic dependent launch: a kernel launched with launch_dependent() may start while the
// kernel before it on the stream drains; what it must not do before pdl_wait() is touch memory that
// kernel writes.  A kernel calls pdl_launch_dependents() once its CTAs are placed.  Both are no-ops
// outside such a pair.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename Args>
static inline cudaError_t launch_dependent(void (*kern)(Args), dim3 grid, int threads, int smem, cudaStream_t st,
                                           const Args &a)
{
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, a);
}

// The segment that holds entry `pos` (largest s with segPtr[s] <= pos; segPtr[0] <= pos), found by one
// warp that probes 32 pointers per step.  The first step looks where even rows would put it, which
// ends the search there for matrices without long rows; otherwise 3 more dependent loads for 20 K
// segments, 4 for a million.
__device__ __forceinline__ int find_segment(const int32_t *segPtr, int64_t n_seg, int64_t first, int64_t end, int64_t pos,
                                            int lane)
{
    int64_t lo = 0, hi = n_seg;
    if (n_seg > 32) {
        int64_t g = (int64_t)((float)(pos - first) / (float)(end - first) * (float)n_seg) - 16;
        g = g < 0 ? 0 : (g > n_seg - 32 ? n_seg - 32 : g);
        const int c = __popc(__ballot_sync(PSPMM_FULL_MASK, __ldg(segPtr + g + lane) <= pos));
        if (c == 32)
            lo = g + 31;
        else if (c == 0)
            hi = g;
        else
            return (int)(g + c - 1);
    }
    while (hi - lo > 1) {
        const int64_t step = (hi - lo + 31) / 32;
        const int64_t p = lo + lane * step;
        const bool ok = p < hi && __ldg(segPtr + p) <= pos;
        const int c = __popc(__ballot_sync(PSPMM_FULL_MASK, ok));
        lo += (int64_t)(c > 0 ? c - 1 : 0) * step;
        hi = lo + step < hi ? lo + step : hi;
    }
    return (int)lo;
}

// Long rows of an unsplit layout, see long_rows.cuh.
#define PSPMM_LONG_ROW 64      // longer rows are cut; one staging window, four batches of 16
#define PSPMM_LONG_ROWS 512    // rows per total, and per look of a share
#define PSPMM_LONG_LOOK 512    // what a look costs, in entries (3 us, at 170 - 250 entries per us and CTA)

struct LongArgs {
    int32_t *totals;    // long rows' entries per PSPMM_LONG_ROWS rows, or nullptr: rows are not cut
    int32_t n_totals;
    int32_t scan_ctas;  // leading CTAs of the first kernel, 8 totals each
    int32_t *counters;  // per share and column tile: partial results that are in, of the row that starts there
    int32_t n_counters;
    float *partials;    // two rows per share
    int32_t shares;     // CTAs (per column tile) of the second kernel
    int32_t own_totals; // 1: these add up the totals themselves (n_totals <= PSPMM_OWN_TOTALS) and need not wait for the first
};
#define PSPMM_OWN_TOTALS 64
#define PSPMM_OWN_ENTRIES 2048  // per SM and share of it, up to which they do

// Host side: sizes for `sms` SMs with `per_sm` resident CTAs of the second kernel: one wave of shares, more
// when they would exceed 16 K entries (equal shares do not end together).
static inline void long_layout(LongArgs *a, int64_t n_rows, int64_t n_entries, int sms, int per_sm, int tiles)
{
    a->n_totals = (int32_t)((n_rows + PSPMM_LONG_ROWS - 1) / PSPMM_LONG_ROWS);
    a->scan_ctas = (a->n_totals + 7) / 8;
    int waves = (int)(n_entries / 16384 / (sms * per_sm)) + 1;
    waves = waves < 16 ? waves : 16;
    a->shares = sms * per_sm > tiles ? sms * per_sm * waves / tiles : 1;
    a->n_counters = a->shares * tiles;
    a->own_totals = 0;
}
// Positions (long_rows.cuh) per share.
__host__ __device__ static inline int64_t long_share_size(int64_t units, int shares)
{
    return ((units + shares - 1) / shares + 63) / 64 * 64;
}
// Whether a share's entries can be counted in an int with room for the groups' spans: only a product so wide
// that its column tiles leave one or two shares fails this.
static inline bool long_fits(const LongArgs &a, int64_t n_entries)
{
    return long_share_size(n_entries + (int64_t)a.n_totals * PSPMM_LONG_LOOK, a.shares) <= 1 << 30;
}
static inline size_t long_head_bytes(const LongArgs &a)
{
    return (((size_t)a.n_totals + (size_t)a.n_counters) * 4 + 255) / 256 * 256;
}
static inline void long_place(LongArgs *a, void *scratch)
{
    a->totals = (int32_t *)scratch;
    a->counters = a->totals + a->n_totals;
    a->partials = (float *)((char *)scratch + long_head_bytes(*a));
}

// One launch of the segment SpMM kernel.  A "segment" is a CSR row, a PCSR row piece, or
// the block-row forms of either.
struct SpmmArgs {
    const int32_t *segPtr;      // [n_seg + 1] entry ranges
    const int32_t *target_row;  // [n_seg] output (block-)row of each segment, or nullptr: row == segment
    const int32_t *colIdx;      // [n_entries]
    const float *val;           // [n_entries * V]
    const float *B;
    float *C;
    int64_t n_seg;
    int64_t n_out;              // output (block-)rows
    int64_t ldB, ldC;
    int32_t nvec;               // dim / VW: vectors per dense row
    int32_t rows_per_group;
    float keep_fraction;        // share of B's lines marked evict-last in L2 (0..1]
    int32_t bucketed;           // target_row carries PSPMM_SEG_* flags, segments come in any order
};

// The kernels that cut long rows get this one.  (Apart, because the register allocation of the others
// changes with the size of their argument.)
struct SpmmLongArgs : SpmmArgs {
    LongArgs lng;  // unsplit layouts: how long rows are cut (totals == nullptr: they are not)
    bool dependent;  // (host) the launch may start while the pre-pass runs
};

// Operands whose width is no multiple of 4: B's rows are padded to 16 bytes, C's are not (spmm_ragged.cu).
struct SpmmRaggedArgs : SpmmLongArgs {
    int32_t dim;  // columns of C; nvec counts the padded ones
};

// Flags in target_row of a length-bucketed plan (pspmm_cfg.bucketed): the low 30 bits are the row.
#define PSPMM_SEG_MULTI 0x80000000u  // the row is cut into several segments: every one of them adds with REDs
#define PSPMM_SEG_FIRST 0x40000000u  // the first of them: the pre-pass zeroes the row when it meets this one
#define PSPMM_SEG_ROW_MASK 0x3fffffffu

struct SddmmArgs {
    const int32_t *segPtr;
    const int32_t *target_row;
    const int32_t *colIdx;
    const float *val;  // mask for V > 1, unused for V == 1
    const float *A;
    const float *B;
    float *out;
    int64_t n_seg;
    int64_t n_rows_A;  // rows of A that exist: block forms read rows arow*V + w only below this
    int64_t ldA, ldB;
    int32_t nvec;
    int32_t rows_per_group;
    float keep_fraction;
    int32_t long_row;    // unsplit rows with more entries are dealt to the first long_ctas CTAs (INT32_MAX: none are)
    int32_t long_range;  // entries per range of those CTAs
    uint32_t long_ctas;
};

// Resolved launch shape.
struct LaunchShape {
    int lpr, vw, cf, threads, rpg, tiles, mlp;
};

// Per-translation-unit dispatchers (one per vector width so the files compile in parallel).
// Return false when (lpr, cf, V) is not instantiated for that width.
bool pspmm_launch_spmm_vw4(const LaunchShape &s, int V, const SpmmLongArgs &a, dim3 grid, cudaStream_t st);
bool pspmm_launch_spmm_vw4_acc(const LaunchShape &s, const SpmmLongArgs &a, dim3 grid, cudaStream_t st);
bool pspmm_launch_spmm_ragged(const LaunchShape &s, const SpmmRaggedArgs &a, dim3 grid, cudaStream_t st);
bool pspmm_launch_spmm_vw2(const LaunchShape &s, int V, const SpmmLongArgs &a, dim3 grid, cudaStream_t st);
bool pspmm_launch_spmm_vw1(const LaunchShape &s, int V, const SpmmLongArgs &a, dim3 grid, cudaStream_t st);
bool pspmm_launch_sddmm_vw4(const LaunchShape &s, int V, const SddmmArgs &a, dim3 grid, cudaStream_t st);
bool pspmm_launch_sddmm_vw2(const LaunchShape &s, int V, const SddmmArgs &a, dim3 grid, cudaStream_t st);
bool pspmm_launch_sddmm_vw1(const LaunchShape &s, int V, const SddmmArgs &a, dim3 grid, cudaStream_t st);

// Smallest instantiated coarsening factor >= need (0 when none).
static inline int pspmm_round_cf(int need)
{
    static const int have[] = {1, 2, 3, 4, 6, 8};
    for (int c : have)
        if (c >= need)
            return c;
    return 0;
}

int pspmm_sm_count();  // of the current device
// Lanes per row of spmm_long_rows_kernel (its column tiles are that many vectors wide).
static inline int pspmm_long_lanes(int nvec, int V) { return nvec > 16 ? 32 : (nvec > 8 || V > 1) ? 16 : (nvec > 4 ? 8 : 4); }
int pspmm_validate_cfg(const pspmm_cfg *cfg, bool sddmm);
enum ShapeUse { SHAPE_ROWS, SHAPE_SPLIT, SHAPE_SDDMM };
// n_seg: (block-)rows or pieces of the layout, negative when they are not known
int pspmm_resolve_shape(const pspmm_cfg *cfg, int32_t dim, int vw_max, int V, ShapeUse use, LaunchShape *out, int64_t n_seg);
int pspmm_vw_max(int32_t dim, int64_t ld0, int64_t ld1, const void *p0, const void *p1);
