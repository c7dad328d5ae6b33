// SpMM whose width is no multiple of 4, on a B with rows padded to 16 bytes: the gathers of the 128-bit family, stores of
// single floats.  (A row of 47 floats admits no wider load than 4 bytes, and the L1 takes a request per row and
// slice: power law of 3.2 M entries, unsplit, 101 columns 210 us, with the copy 144; 255 columns 504 and 271.)
// pad_rows_kernel makes the padded copy; the layers' projections come padded.  Against products of the next multiple of 4 it
// costs up to 9 % on even rows and 3 - 20 % on a power law (stores of single floats, two barriers per row: 100 K rows of 32, 101 columns 103 and
// 98 us, split power law of it, 47 columns 79 and 66), and saves them the pass that cuts the result back.
#include "spmm_kernel.cuh"

#define CFS(LPR_) \
    PSPMM_SPMM_CASE_RAGGED(LPR_, 1) PSPMM_SPMM_CASE_RAGGED(LPR_, 2) PSPMM_SPMM_CASE_RAGGED(LPR_, 3) PSPMM_SPMM_CASE_RAGGED(LPR_, 4)

static bool launch_segments(const LaunchShape &s, const SpmmRaggedArgs &a, dim3 grid, cudaStream_t st)
{
    CFS(4)
    CFS(8)
    CFS(16)
    CFS(32)
    return false;
}

bool pspmm_launch_spmm_ragged(const LaunchShape &s, const SpmmRaggedArgs &a, dim3 grid, cudaStream_t st)
{
    if (!launch_segments(s, a, grid, st))
        return false;
    if (a.lng.totals)
        spmm_launch_long_rows<4, 1, true>(a, st);
    return true;
}

// dst row i = the dim floats of src row i and zeros up to the next multiple of 4.  Bound: HBM or L2 (one read, one
// write); four vectors per thread.
__global__ void __launch_bounds__(256) pad_rows_kernel(const float *__restrict__ src, float *__restrict__ dst, int64_t n,
                                                       int dim, int64_t ld_src, int64_t ld_dst)
{
    const int nvec = (dim + 3) / 4;
    const int64_t total = n * nvec, stride = (int64_t)gridDim.x * 256;
    for (int64_t t0 = (int64_t)blockIdx.x * 256 + threadIdx.x; t0 < total; t0 += 4 * stride) {
        float v[4][4];
        int64_t row[4];
        int col[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t t = t0 + u * stride;
            // (a 64-bit division is a call; most operands have fewer than 2^32 vectors)
            row[u] = total <= UINT32_MAX ? (int64_t)((uint32_t)t / (uint32_t)nvec) : t / nvec;
            col[u] = (int)(t - row[u] * nvec) * 4;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                v[u][i] = t < total && col[u] + i < dim ? __ldg(src + row[u] * ld_src + col[u] + i) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (t0 + u * stride < total)
                *reinterpret_cast<float4 *>(dst + row[u] * ld_dst + col[u]) = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
    }
}

extern "C" int pspmm_pad_rows(const float *src, float *dst, int64_t n, int32_t dim, int64_t ld_src, int64_t ld_dst,
                              void *stream)
{
    if (n < 0 || dim <= 0 || ld_src < dim || ld_dst < dim || ld_dst % 4 != 0 || (uintptr_t)dst % 16 != 0)
        return PSPMM_E_ARG;
    if (n == 0)
        return PSPMM_OK;
    if (!src || !dst)
        return PSPMM_E_ARG;
    const int64_t ctas = (n * ((dim + 3) / 4) + 1023) / 1024, most = (int64_t)pspmm_sm_count() * 32;
    pad_rows_kernel<<<(unsigned)(ctas < most ? ctas : most), 256, 0, (cudaStream_t)stream>>>(src, dst, n, dim, ld_src, ld_dst);
    PSPMM_CUDA_TRY(cudaGetLastError());
    return PSPMM_OK;
}
