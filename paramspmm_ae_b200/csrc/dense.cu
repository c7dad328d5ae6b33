// Dense fp32 products of the layers on the 5th-generation tensor cores (sm_100a):
//
//     C[M, N] = op(A) op(B),   fp32 in, fp32 out, fp32 accuracy.
//
// The layers multiply tall node matrices by small weights: H W and G W^T (M = nodes, N and K = layer
// widths) and H^T G (K = nodes).  CUDA cores give these 40 - 46 TFLOP/s (a third of a full-size GCN
// training step).  Here every operand value is split in registers into three bf16 parts,
//     x = h + m + l   (h = rn(x), m = rn(x - h), l = x - h - m: 8 + 8 + 8 bits, nothing is lost),
// and six of the nine products run as tcgen05.mma kind::f16 with fp32 accumulation in TMEM:
// h h, h m, m h, m m, h l, l h.  The three left out are below 2^-26 of the product, less than the
// rounding of one fp32 multiply-add.
//
// Accumulation.  tcgen05.mma truncates when it adds to the accumulator (measured: 1 + 15 x 0.75 ulp
// over separate k-steps stays 1), so a long chain of them is biased: K = 4096 in one chain is 20 x
// less accurate than an fp32 FMA chain.  A chain here is one stage of 32 k: the five small products
// of its two k-steps first, while the accumulator is below 2^-8 of its final size, then the two h h,
// so two truncations at full size per chain; the chains are summed in registers with round-to-nearest
// fp32 adds.
//
// Structure: one persistent CTA per SM, a ring of three stages.  Three groups of four warps own one slot
// of the ring each: a group fetches the fp32 tiles of its next stage, splits them and writes A's bf16
// parts to TMEM (a lane per row, so the MMA reads A from there) and B's to shared memory (K-major core
// matrices without swizzle: 8 consecutive rows of 16 bytes, so the 16-byte stores of neighbouring
// lanes never conflict).  A and, where both are contiguous along M and N, B pass through raw tiles in
// shared memory (cp.async, padded rows), from which each lane takes its row of A and its chunks of B.
// Two warps issue the MMAs; eight add finished chains out of TMEM (two buffers of 128 columns) into
// registers and store the tile.  B of the tall products, the weights, is the same for every row tile:
// split_weights_kernel splits it once into caller scratch, in the layout of the stages, and one warp
// brings its tiles in with bulk copies.  Products with a long K are cut into splits whose partial
// tiles are summed by reduce_splits_kernel.
//
// What the shape rests on (2.4 M x 256 x 256; cuBLAS 5.6 ms).  All loading warps on one stage at a time
// waited out a memory latency per stage however far ahead they loaded (a warp's scoreboard does not
// tell one batch of loads from the next): 3.6 ms; independent groups: 2.7 ms, then bound by shared
// memory, 8 KB of operands per 64-clock MMA; A in TMEM halves that and saves its stores.
//
// Infinities, NaNs and values that round to infinity in bf16 have no such split: a CTA that meets one
// computes its tiles with fp32 FMAs from then on.
//
// Every wait is bounded (about two seconds).  When one runs out the CTA raises g_dense_status, which
// pspmm_dense_status reads, fills what it has not computed of C with NaN, and leaves.
#include <type_traits>

#include "pspmm_common.cuh"

namespace {

constexpr int BM = 128, BN = 128, BK = 32;
constexpr int STAGES = 3, ACC_BUFS = 2;
constexpr int PLANE = BN * BK * 2;               // one bf16 tile of B
constexpr int STAGE_BYTES = 3 * PLANE;
constexpr int RAW_PITCH = BK + 4;                // floats per row of a raw tile of k-contiguous A
constexpr int RAW_PITCH_T = 128 + 4;             // floats per k of a raw tile that is contiguous along M or N
constexpr int RAW_BYTES = BM * RAW_PITCH * 4;
constexpr int RAW_BYTES_T = BK * RAW_PITCH_T * 4;
constexpr int OUT_PITCH = 36;                    // floats per row of a drainer's 32 x 32 output patch
constexpr int OUT_BYTES = 32 * OUT_PITCH * 4;
constexpr int TMEM_A = ACC_BUFS * BN;            // first column of A's parts: 16 columns per part and stage
constexpr int TMEM_COLS = 512;
constexpr int GROUP_WARPS = 4, LOADERS = STAGES * GROUP_WARPS, DRAINERS = 8;
constexpr int MMA_WARP = LOADERS + DRAINERS, BULK_WARP = MMA_WARP + 1;
constexpr int THREADS = (LOADERS + DRAINERS + 4) * 32;
// Registers per thread after the split: 768 x 80 = 61,440 at launch; 384 x 80 + 256 x 104 + 128 x 32 = 61,440.
constexpr int DRAINER_REGS = 104, OTHER_REGS = 32;

// Raw tiles of one slot: k-contiguous A, or A and B that are both contiguous the other way.
template <bool KC_A, bool KC_B, bool PRE>
struct Raw {
    static constexpr bool BOTH = !PRE && !KC_A && !KC_B;
    static constexpr int BYTES = KC_A ? RAW_BYTES : (BOTH ? 2 * RAW_BYTES_T : 0);
    static constexpr int SMEM = STAGES * (STAGE_BYTES + BYTES) + DRAINERS * OUT_BYTES + 1024;
};


__device__ unsigned g_dense_status;

struct DenseArgs {
    const float *A, *B;
    float *C;                 // output, or partial tiles [splits][M][N] when splits > 1
    int64_t ldA, ldB, ldC;
    int32_t M, N, K;
    int32_t k_per_split;      // a multiple of BK
    int32_t splits, m_tiles, n_tiles, bn;  // bn: columns per tile, a multiple of 16
    int32_t vecA, vecB;       // k-contiguous operands: rows may be read 16 bytes at a time
    const unsigned char *Bs;  // B split beforehand (split_weights_kernel)
    unsigned *odd;            // with Bs: one word per block of that kernel, set when a value of B has no split
    int32_t odd_words;
    uint32_t wait_ns;         // limit of a wait
    int32_t withhold;         // arrivals that no one brings: 0, or 1 to make the waits for a stage run out
};

struct ReduceArgs {
    const float *part;
    float *C;
    int64_t ldC;
    int32_t splits, M, N;
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint32_t bar, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool bar_try(uint32_t bar, int parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 0x989680;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// False when the wait ran out (or another role's did: *abort).  Whole warps call it, and its lanes agree: what
// follows are barriers and tcgen05 instructions of whole warps.
__device__ __forceinline__ bool bar_wait(uint32_t bar, int parity, volatile int *abort, uint32_t limit_ns)
{
    if (__all_sync(PSPMM_FULL_MASK, bar_try(bar, parity)))
        return true;
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    while (!__all_sync(PSPMM_FULL_MASK, bar_try(bar, parity))) {
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        if (__any_sync(PSPMM_FULL_MASK, *abort || t - t0 > limit_ns)) {
            *abort = 1;
            atomicExch(&g_dense_status, 1u);
            return false;
        }
    }
    return true;
}

// Descriptor of a K-major tile without swizzle: 8-row groups 128 bytes apart, 16-byte k-chunks
// rows * 16 bytes apart.
__device__ __forceinline__ uint64_t tile_desc(uint32_t addr, int rows)
{
    return (uint64_t)((addr & 0x3ffff) >> 4) | ((uint64_t)rows << 16) | ((uint64_t)(128 >> 4) << 32) | (1ull << 46);
}

// A in TMEM, B in shared memory.
__device__ __forceinline__ void mma(uint32_t acc, uint32_t a, uint64_t b, uint32_t idesc, int accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(acc), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ bool elect_one()
{
    uint32_t on;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(on));
    return on != 0;
}
__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// Eight accumulator columns of the warp's 32 TMEM lanes; complete after tcgen05.wait::ld.
__device__ __forceinline__ void acc_load(uint32_t (&v)[8], uint32_t addr)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(addr));
}

// Two values -> their bf16 pair (first value in the low half) and what is left of them.
__device__ __forceinline__ uint32_t split_pair(float &x0, float &x1)
{
    uint32_t p;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(x1), "f"(x0));
    x0 -= __uint_as_float(p << 16);
    x1 -= __uint_as_float(p & 0xffff0000u);
    return p;
}

// Eight fp32 values along k of one row -> three 16-byte chunks.  Returns false if a value has no
// split (the remainder of an infinity, a NaN or an overflow is not finite).
__device__ __forceinline__ bool split_store(const float (&x)[8], unsigned char *dst, int plane)
{
    float r[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
        r[i] = x[i];
    uint4 h, m, l;
    h.x = split_pair(r[0], r[1]);
    h.y = split_pair(r[2], r[3]);
    h.z = split_pair(r[4], r[5]);
    h.w = split_pair(r[6], r[7]);
    const float sum = ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
    m.x = split_pair(r[0], r[1]);
    m.y = split_pair(r[2], r[3]);
    m.z = split_pair(r[4], r[5]);
    m.w = split_pair(r[6], r[7]);
    l.x = split_pair(r[0], r[1]);
    l.y = split_pair(r[2], r[3]);
    l.z = split_pair(r[4], r[5]);
    l.w = split_pair(r[6], r[7]);
    *reinterpret_cast<uint4 *>(dst) = h;
    *reinterpret_cast<uint4 *>(dst + plane) = m;
    *reinterpret_cast<uint4 *>(dst + 2 * plane) = l;
    return fabsf(sum) < __int_as_float(0x7f800000);
}

// One part (16 packed columns) of the warp's 32 rows of A -> TMEM.
__device__ __forceinline__ void part_store(uint32_t addr, const uint32_t (&v)[16])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                 "%14, %15, %16};"
                 ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
                 "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}

// The 32 k of a lane's row -> the three parts of a stage.  Returns as split_store.
__device__ __forceinline__ bool split_row(float (&x)[BK], uint32_t addr)
{
    uint32_t v[16];
    float sum[4] = {};
#pragma unroll
    for (int p = 0; p < 3; ++p) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            v[i] = split_pair(x[2 * i], x[2 * i + 1]);
        part_store(addr + p * 16, v);
        if (p == 0) {
#pragma unroll
            for (int i = 0; i < BK; ++i)
                sum[i & 3] += x[i];
        }
    }
    return fabsf((sum[0] + sum[1]) + (sum[2] + sum[3])) < __int_as_float(0x7f800000);
}

// cp.async of `bytes` (0 .. N) out of N; the rest is filled with zeros.
template <int N>
__device__ __forceinline__ void copy_async(uint32_t dst, const float *src, int bytes)
{
    if constexpr (N == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Barrier of one group's 128 threads; true if all bring true.
__device__ __forceinline__ bool group_all(int id, bool ok)
{
    int all;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\t"
                 "barrier.cta.red.and.aligned.pred q, %2, 128, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
                 : "=r"(all) : "r"((int)ok), "r"(id) : "memory");
    return all != 0;
}

// Chunk `idx` of a tile of 128 rows x 32 k: which row and which eight k.  Lanes run along the
// contiguous direction of the source as far as the 16-byte shared-memory stores allow (eight
// neighbouring rows per store phase).
template <bool KC>
__device__ __forceinline__ void chunk_place(int idx, int &row, int &kc)
{
    if constexpr (KC) {
        row = (idx & 7) | ((idx >> 5) << 3);
        kc = (idx >> 3) & 3;
    } else {
        row = idx & 127;
        kc = idx >> 7;
    }
}

// Volatile: the loads of a later stage are to leave before this stage's wait, not at their first use.
__device__ __forceinline__ float4 load4(const float *p)
{
    float4 v;
    asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float load1(const float *p)
{
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// KC: element (r, k) lies at p[r * ld + k]; otherwise at p[k * ld + r].
template <bool KC>
__device__ __forceinline__ void chunk_load_whole(float (&x)[8], const float *p, int64_t ld, int r, int k)
{
    if constexpr (KC) {
        const float4 a = load4(p + (int64_t)r * ld + k), b = load4(p + (int64_t)r * ld + k + 4);
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
        x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
            x[j] = load1(p + (int64_t)(k + j) * ld + r);
    }
}
// The same at the edges: rows and k beyond the ends are zeros, rows may be misaligned.
template <bool KC>
__device__ __forceinline__ void chunk_load(float (&x)[8], const float *p, int64_t ld, int r, int rows, int k, int k_end)
{
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        x[j] = 0.f;
        if (r < rows && k + j < k_end)
            x[j] = load1(KC ? p + (int64_t)r * ld + k + j : p + (int64_t)(k + j) * ld + r);
    }
}

// B split beforehand: tile (n_tile, k_stage) is three planes of [k chunk][bn rows][8 bf16].
template <bool KC_B>
__global__ void __launch_bounds__(256) split_weights_kernel(const DenseArgs a, unsigned char *dst)
{
    pdl_launch_dependents();
    const int64_t k_stages = (a.K + BK - 1) / BK;
    const int64_t total = (int64_t)a.n_tiles * k_stages * a.bn * 4;
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    bool plain = true;
    if (i < total) {
        const int row = (int)(i % a.bn);
        const int kc = (int)(i / a.bn % 4);
        const int64_t tile = i / a.bn / 4;  // n_tile * k_stages + k_stage
        const int n0 = (int)(tile / k_stages) * a.bn, k0 = (int)(tile % k_stages) * BK;
        float x[8];
        chunk_load<KC_B>(x, a.B, a.ldB, n0 + row, n0 + a.bn < a.N ? n0 + a.bn : a.N, k0 + kc * 8, a.K);
        plain = split_store(x, dst + tile * (3 * a.bn * 64) + kc * (a.bn * 16) + row * 16, a.bn * 64);
    }
    const int odd = __syncthreads_or(!plain);
    if (threadIdx.x == 0)
        a.odd[blockIdx.x] = odd ? 1u : 0u;
}

// PRE: B comes split (a.Bs), only A passes through registers.
template <bool KC_A, bool KC_B, bool PRE>
__global__ void __launch_bounds__(THREADS, 1) dense_kernel(const DenseArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[2 * STAGES + 2 * ACC_BUFS];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int abort_flag, odd_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t full = smem_addr(bars), empty = full + 8 * STAGES, acc_full = empty + 8 * STAGES,
                   acc_empty = acc_full + 8 * ACC_BUFS;
    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            bar_init(full + 8 * i, GROUP_WARPS + (PRE ? 1 : 0) + a.withhold);
            bar_init(empty + 8 * i, 1);
        }
        for (int i = 0; i < ACC_BUFS; ++i) {
            bar_init(acc_full + 8 * i, 1);
            bar_init(acc_empty + 8 * i, DRAINERS);
        }
        abort_flag = 0;
        odd_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_addr(&tmem_base)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    const int items = a.m_tiles * a.n_tiles * a.splits;
    pdl_launch_dependents();

    // Work item -> tile and k range; items that share a row tile are neighbours.
    auto item_place = [&](int item, int &m0, int &n0, int &k0, int &k1, int &split) {
        const int nt = item % a.n_tiles;
        item /= a.n_tiles;
        const int mt = item % a.m_tiles;
        split = item / a.m_tiles;
        m0 = mt * BM;
        n0 = nt * a.bn;
        k0 = split * a.k_per_split;
        k1 = a.K - k0 > a.k_per_split ? k0 + a.k_per_split : a.K;
    };

    if (warp < LOADERS) {
        // Group q fills slot q: stages q, q + 4, ... of the CTA's sequence of items.
        const int q = warp / GROUP_WARPS, tid = threadIdx.x % (GROUP_WARPS * 32);
        unsigned char *st = smem + q * STAGE_BYTES;
        int phase = 0;
        int item = blockIdx.x, m0 = 0, n0 = 0, k0 = 0, k1 = 0, split, len = 0, j = q;
        auto settle = [&]() {  // j stages into `item` -> the item it lies in
            while (item < items) {
                item_place(item, m0, n0, k0, k1, split);
                len = (k1 - k0 + BK - 1) / BK;
                if (j < len)
                    break;
                j -= len;
                item += gridDim.x;
            }
        };
        settle();
        const int row = tid;  // of the tile, as the TMEM lanes have it
        const uint32_t parts = tmem + ((uint32_t)((warp & 3) * 32) << 16) + TMEM_A + q * 48;
        float *raw = reinterpret_cast<float *>(smem + STAGES * STAGE_BYTES + q * Raw<KC_A, KC_B, PRE>::BYTES);
        float x[BK];
        auto fetch_raw = [&]() {  // k-contiguous A
            const int k = k0 + j * BK, left = k1 - k;
            if (a.vecA) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = (tid >> 3) + i * 16, c = (tid & 7) * 4;
                    int n = m0 + r < a.M ? left - c : 0;
                    n = n < 0 ? 0 : (n > 4 ? 4 : n);
                    copy_async<16>(smem_addr(raw + r * RAW_PITCH + c), a.A + (n ? (int64_t)(m0 + r) * a.ldA + k + c : 0),
                                   n * 4);
                }
            } else {
                for (int i = 0; i < 32; ++i) {
                    const int r = (tid >> 5) + i * 4, c = tid & 31;
                    const int n = m0 + r < a.M && c < left ? 1 : 0;
                    copy_async<4>(smem_addr(raw + r * RAW_PITCH + c), a.A + (n ? (int64_t)(m0 + r) * a.ldA + k + c : 0),
                                  n * 4);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        // Tiles that are contiguous along M or N: [k][128]
        constexpr bool BOTH = Raw<KC_A, KC_B, PRE>::BOTH;
        float *raw_b = raw + BK * RAW_PITCH_T;
        auto fetch_raw_t = [&](float *dst, const float *p, int64_t ld, int c0, int c_end, bool aligned, int k, int k_end) {
            if (aligned) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int kr = (tid >> 5) + i * 4, c = (tid & 31) * 4;
                    int n = k + kr < k_end ? c_end - (c0 + c) : 0;
                    n = n < 0 ? 0 : (n > 4 ? 4 : n);
                    copy_async<16>(smem_addr(dst + kr * RAW_PITCH_T + c), p + (n ? (int64_t)(k + kr) * ld + c0 + c : 0), n * 4);
                }
            } else {
                for (int kr = 0; kr < BK; ++kr) {
                    const int n = k + kr < k_end && c0 + tid < c_end ? 1 : 0;
                    copy_async<4>(smem_addr(dst + kr * RAW_PITCH_T + tid), p + (n ? (int64_t)(k + kr) * ld + c0 + tid : 0),
                                  n * 4);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        auto fetch_a_t = [&]() { fetch_raw_t(raw, a.A, a.ldA, m0, a.M, a.vecA, k0 + j * BK, k1); };
        auto fetch_b_t = [&]() {
            fetch_raw_t(raw_b, a.B, a.ldB, n0, n0 + a.bn < a.N ? n0 + a.bn : a.N, a.vecB, k0 + j * BK, k1);
        };
        auto fetch_columns = [&]() {  // A contiguous along M
            const int k = k0 + j * BK;
            const bool in = m0 + row < a.M;
            const float *p = a.A + (in ? (int64_t)k * a.ldA + m0 + row : 0);
            if (k + BK <= k1 && m0 + BM <= a.M) {
#pragma unroll
                for (int i = 0; i < BK; ++i)
                    x[i] = load1(p + (int64_t)i * a.ldA);
            } else {
#pragma unroll
                for (int i = 0; i < BK; ++i) {
                    x[i] = 0.f;
                    if (in && k + i < k1)
                        x[i] = load1(p + (int64_t)i * a.ldA);
                }
            }
        };
        if (item < items) {
            if constexpr (KC_A) {
                fetch_raw();
            } else if constexpr (BOTH) {
                fetch_a_t();
                fetch_b_t();
            } else {
                fetch_columns();
            }
        }
        bool ok = true;
        while (item < items) {
            const int k_now = k0 + j * BK, k1_now = k1, n0_now = n0;
            j += STAGES;
            if constexpr (KC_A) {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                if (!group_all(1 + q, ok))
                    break;
#pragma unroll
                for (int i = 0; i < BK / 4; ++i) {
                    const float4 v = *reinterpret_cast<const float4 *>(raw + row * RAW_PITCH + 4 * i);
                    x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
                }
                group_all(1 + q, true);
                settle();
                if (item < items)
                    fetch_raw();
            } else if constexpr (BOTH) {
                // Each next fetch leaves as soon as its tile has been read, so that it is in flight while
                // this stage is split.
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                if (!group_all(1 + q, ok))
                    break;
#pragma unroll
                for (int i = 0; i < BK; ++i)
                    x[i] = raw[i * RAW_PITCH_T + row];
                group_all(1 + q, true);
                settle();
                if (item < items)
                    fetch_a_t();
            } else {
                settle();
            }
            ok = bar_wait(empty + 8 * q, phase ^ 1, &abort_flag, a.wait_ns);
            if (!ok) {
                if constexpr (BOTH)
                    group_all(1 + q, true);  // (warps of the group that saw the stage free are at this barrier below)
                if constexpr (KC_A || BOTH)
                    continue;  // (the group leaves together)
                else
                    break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            bool plain = true;
            if constexpr (BOTH) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    int r, kc;
                    chunk_place<false>(tid + i * (GROUP_WARPS * 32), r, kc);
                    if (r < a.bn) {
                        float y[8];
#pragma unroll
                        for (int t = 0; t < 8; ++t)
                            y[t] = raw_b[(kc * 8 + t) * RAW_PITCH_T + r];
                        plain &= split_store(y, st + kc * (a.bn * 16) + r * 16, PLANE);
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                group_all(1 + q, true);
                if (item < items)
                    fetch_b_t();
            } else if constexpr (!PRE) {
                const int n_end = n0_now + a.bn < a.N ? n0_now + a.bn : a.N;
                const bool whole = k_now + BK <= k1_now && n0_now + BN <= n_end && (!KC_B || a.vecB);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    int r, kc;
                    chunk_place<KC_B>(tid + i * (GROUP_WARPS * 32), r, kc);
                    float y[8];
                    if (whole)
                        chunk_load_whole<KC_B>(y, a.B, a.ldB, n0_now + r, k_now + kc * 8);
                    else
                        chunk_load<KC_B>(y, a.B, a.ldB, n0_now + r, n_end, k_now + kc * 8, k1_now);
                    if (r < a.bn)
                        plain &= split_store(y, st + kc * (a.bn * 16) + r * 16, PLANE);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            plain &= split_row(x, parts);
            if (!plain)
                odd_flag = 1;
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                bar_arrive(full + 8 * q);
            phase ^= 1;
            if constexpr (!KC_A && !BOTH) {
                if (item < items)
                    fetch_columns();
            }
        }
        if constexpr (KC_A || BOTH)
            asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else if (warp >= MMA_WARP) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(OTHER_REGS));
        if (PRE && warp == BULK_WARP) {
            pdl_wait();  // split_weights_kernel writes what is copied here
            for (int i = lane; i < a.odd_words; i += 32)
                if (*(volatile unsigned *)(a.odd + i))
                    odd_flag = 1;
            __syncwarp();
            const int k_stages = (a.K + BK - 1) / BK;
            const int plane = a.bn * 64;
            int stage = 0, phase = 0;
            bool ok = true;
            for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
                int m0, n0, k0, k1;
                int split;
                item_place(item, m0, n0, k0, k1, split);
                const unsigned char *src = a.Bs + (int64_t)(n0 / a.bn * k_stages + k0 / BK) * (3 * plane);
                for (int k = k0; k < k1; k += BK, src += 3 * plane) {
                    if (!bar_wait(empty + 8 * stage, phase ^ 1, &abort_flag, a.wait_ns)) {
                        ok = false;
                        break;
                    }
                    if (lane == 0) {
                        const uint32_t bar = full + 8 * stage;
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(3 * plane) : "memory");
                        const uint32_t st = smem_addr(smem) + stage * STAGE_BYTES;
#pragma unroll
                        for (int p = 0; p < 3; ++p)
                            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                         ::"r"(st + p * PLANE), "l"(src + p * plane), "r"(plane), "r"(bar) : "memory");
                    }
                    __syncwarp();
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
        }
        if (warp == MMA_WARP || warp == MMA_WARP + 2) {
            // Two warps issue, a chain (stage) each in turn: one warp's waits, twelve issues and commits
            // (1,600 clocks) would outlast the MMAs (800).
            const int m = warp == MMA_WARP ? 0 : 1;  // also the accumulator buffer
            // D fp32, A and B bf16, both K-major
            const uint32_t idesc =
                (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(a.bn >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
            const uint32_t acc = tmem + m * BN;
            const uint64_t desc0 = tile_desc(smem_addr(smem), a.bn);
            int stage = 0, phase = 0, i = 0;
            bool ok = true;
            for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
                int m0, n0, k0, k1;
                int split;
                item_place(item, m0, n0, k0, k1, split);
                for (int k = k0; k < k1; k += BK, ++i) {
                    if ((i & 1) == m) {
                        if (!bar_wait(acc_empty + 8 * m, ((i >> 1) & 1) ^ 1, &abort_flag, a.wait_ns) ||
                            !bar_wait(full + 8 * stage, phase, &abort_flag, a.wait_ns)) {
                            ok = false;
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        if (elect_one()) {
                            const uint32_t pa = tmem + TMEM_A + stage * 48;
                            const uint64_t pb = desc0 + (uint64_t)(stage * (STAGE_BYTES >> 4));
                            // product p: which part of A and which of B; the two h h of the stage come last
                            constexpr int PA[6] = {1, 2, 0, 1, 0, 0}, PB[6] = {1, 0, 2, 0, 1, 0};
#pragma unroll
                            for (int p = 0; p < 6; ++p)
#pragma unroll
                                for (int s = 0; s < BK / 16; ++s)
                                    mma(acc, pa + PA[p] * 16 + s * 8,
                                        pb + (uint64_t)(PB[p] * (PLANE >> 4) + s * 2 * a.bn), idesc, p + s > 0);
                            mma_commit(empty + 8 * stage);
                            mma_commit(acc_full + 8 * m);
                        }
                        __syncwarp();
                    }
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(DRAINER_REGS));
        // Drainer d: TMEM lanes (rows) of its quadrant, half the columns.
        const int d = warp - LOADERS;
        const int quad = warp & 3, half = d >> 2;
        const int row = quad * 32 + lane;
        const int cols = a.bn / 2;  // a multiple of 8
        float *patch = reinterpret_cast<float *>(smem + STAGES * (STAGE_BYTES + Raw<KC_A, KC_B, PRE>::BYTES) + d * OUT_BYTES);
        int buf = 0, buf_phase = 0;
        bool ok = true;
        int item = blockIdx.x;
        for (; item < items; item += gridDim.x) {
            int m0, n0, k0, k1;
            int split;
            item_place(item, m0, n0, k0, k1, split);
            float acc[64];
#pragma unroll
            for (int j = 0; j < 64; ++j)
                acc[j] = 0.f;
            for (int k = k0; k < k1; k += BK) {
                if (!bar_wait(acc_full + 8 * buf, buf_phase, &abort_flag, a.wait_ns)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int q0 = 0; q0 < 8; q0 += 4) {
                    if (q0 * 8 >= cols)
                        break;
                    uint32_t v[4][8];
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if ((q0 + q) * 8 < cols)
                            acc_load(v[q], tmem + ((uint32_t)(quad * 32) << 16) + buf * BN + half * cols + (q0 + q) * 8);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if ((q0 + q) * 8 < cols)
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                asm volatile("" : "+r"(v[q][j]));  // (not read ahead of the wait)
                                acc[(q0 + q) * 8 + j] += __uint_as_float(v[q][j]);
                            }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0)
                    bar_arrive(acc_empty + 8 * buf);
                if (++buf == ACC_BUFS) {
                    buf = 0;
                    buf_phase ^= 1;
                }
            }
            if (!ok)
                break;
            const int c0 = n0 + half * cols;
            const int c1 = n0 + a.bn < a.N ? n0 + a.bn : a.N;
            float *out = a.C + ((int64_t)split * a.M + m0 + quad * 32) * a.ldC + c0;
            const int rows = a.M - m0 - quad * 32;  // of the warp's 32
            if (odd_flag) {  // some operand value has no bf16 split
                const int r = m0 + row;
                for (int j = 0; lane < rows && j < cols && c0 + j < c1; ++j) {
                    float s = 0.f;
                    for (int k = k0; k < k1; ++k)
                        s = fmaf(KC_A ? a.A[(int64_t)r * a.ldA + k] : a.A[(int64_t)k * a.ldA + r],
                                 KC_B ? a.B[(int64_t)(c0 + j) * a.ldB + k] : a.B[(int64_t)k * a.ldB + c0 + j], s);
                    out[lane * a.ldC + j] = s;
                }
                continue;
            }
            // 32 columns at a time through shared memory, so that eight lanes store 128 bytes of a row (a
            // lane per row would touch 32 lines per store: 6,900 clocks per tile).
            const bool vec = (a.ldC & 3) == 0 && ((uintptr_t)out & 15) == 0;
#pragma unroll
            for (int j0 = 0; j0 < 64; j0 += 32) {
                if (j0 >= cols)
                    break;
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    *reinterpret_cast<float4 *>(patch + lane * OUT_PITCH + j) =
                        make_float4(acc[j0 + j], acc[j0 + j + 1], acc[j0 + j + 2], acc[j0 + j + 3]);
                __syncwarp();
                if (vec) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int r = (lane >> 3) + i * 4, c = (lane & 7) * 4;
                        const float4 v = *reinterpret_cast<const float4 *>(patch + r * OUT_PITCH + c);
                        float *o = out + r * a.ldC + j0 + c;
                        const int left = j0 + c < cols ? c1 - (c0 + j0 + c) : 0;
                        if (r < rows) {
                            if (left >= 4) {
                                *reinterpret_cast<float4 *>(o) = v;
                            } else {
                                if (left > 0)
                                    o[0] = v.x;
                                if (left > 1)
                                    o[1] = v.y;
                                if (left > 2)
                                    o[2] = v.z;
                            }
                        }
                    }
                } else {
                    for (int r = 0; r < 32 && r < rows; ++r)
                        if (j0 + lane < cols && c0 + j0 + lane < c1)
                            out[r * a.ldC + j0 + lane] = patch[r * OUT_PITCH + lane];
                }
            }
        }
        for (; item < items; item += gridDim.x) {  // a wait ran out: no stale memory passes for a result
            int m0, n0, k0, k1;
            int split;
            item_place(item, m0, n0, k0, k1, split);
            const int c0 = n0 + half * cols;
            const int c1 = n0 + a.bn < a.N ? n0 + a.bn : a.N;
            if (m0 + row < a.M)
                for (int c = c0; c < c0 + cols && c < c1; ++c)
                    a.C[((int64_t)split * a.M + m0 + row) * a.ldC + c] = __int_as_float(0x7fffffff);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == MMA_WARP && abort_flag) {  // let the MMAs in flight end (they wait on nothing)
        for (int i = 0; i < 1000; ++i)
            __nanosleep(1000);
    }
    if (warp == MMA_WARP)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
}

// C = sum of the partial tiles: a block takes 32 neighbouring elements, its eight warps the splits in
// turn (one thread per element walking 148 splits took 9 us of a 31 us product).
__global__ void __launch_bounds__(256) reduce_splits_kernel(const ReduceArgs a)
{
    __shared__ float sums[8][33];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t total = (int64_t)a.M * a.N;
    const int64_t i = (int64_t)blockIdx.x * 32 + lane;
    pdl_wait();
    float s[4] = {};
    if (i < total) {
        int t = warp;
        for (; t + 24 < a.splits; t += 32)
#pragma unroll
            for (int u = 0; u < 4; ++u)
                s[u] += a.part[(t + 8 * u) * total + i];
        for (; t < a.splits; t += 8)
            s[0] += a.part[t * total + i];
    }
    sums[warp][lane] = (s[0] + s[1]) + (s[2] + s[3]);
    __syncthreads();
    if (warp == 0 && i < total) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w)
            t += sums[w][lane];
        a.C[i / a.N * a.ldC + i % a.N] = t;
    }
}

// Tiles and splits of a product.  The persistent CTAs take the items in turn, so a launch lasts
// (rounds) x (stages per item + start and end of a tile, about 6 stages' time); cutting K evens out the
// rounds and gives every SM an item, and costs the partial tiles' trip through memory (a stage lasts
// about 0.7 us, in which the chip moves 2 MB of them) and one more launch (5 stages' time).
void plan(int64_t M, int64_t N, int64_t K, DenseArgs &a)
{
    a.m_tiles = (int32_t)((M + BM - 1) / BM);
    a.n_tiles = (int32_t)((N + BN - 1) / BN);
    const int64_t per = (N + a.n_tiles - 1) / a.n_tiles;
    a.bn = (int32_t)((per + 15) / 16 * 16);
    const int64_t tiles = (int64_t)a.m_tiles * a.n_tiles, sms = pspmm_sm_count();
    const int64_t stages = (K + BK - 1) / BK;
    a.splits = 1;
    a.k_per_split = (int32_t)(stages * BK);
    if (tiles >= 8 * sms)
        return;  // enough rounds
    double best = 1e30;
    for (int64_t rounds = 0; rounds <= 8; ++rounds) {
        int64_t splits = rounds * sms / tiles;  // (0 rounds: no split)
        splits = splits < 1 ? 1 : (splits > stages ? stages : splits);
        const int64_t len = (stages + splits - 1) / splits;
        splits = (stages + len - 1) / len;
        double cost = (double)((tiles * splits + sms - 1) / sms) * (double)(len + 6);
        if (splits > 1)
            cost += 5 + (double)splits * (double)M * (double)N * 8.0 / 2e6;
        if (cost < best) {
            best = cost;
            a.splits = (int32_t)splits;
            a.k_per_split = (int32_t)(len * BK);
        }
    }
}

// The weights are worth splitting beforehand when many row tiles use them and a CTA goes through more
// than a few stages (19,717 x 16 x 500: 25 us against 46; 19,717 x 16 x 3: 9.1 against 8.3).
bool presplit(const DenseArgs &a)
{
    const int64_t rounds = ((int64_t)a.m_tiles * a.n_tiles * a.splits + pspmm_sm_count() - 1) / pspmm_sm_count();
    return a.m_tiles >= 16 && rounds * (a.k_per_split / BK) >= 6;
}

size_t partial_bytes(const DenseArgs &a, int64_t M, int64_t N)
{
    return a.splits > 1 ? ((size_t)a.splits * (size_t)M * (size_t)N * sizeof(float) + 255) / 256 * 256 : 0;
}

// Blocks of split_weights_kernel, and the bytes of its verdicts and tiles.
int64_t split_blocks(const DenseArgs &a, int64_t K)
{
    return ((int64_t)a.n_tiles * ((K + BK - 1) / BK) * a.bn * 4 + 255) / 256;
}
size_t odd_bytes(const DenseArgs &a, int64_t K) { return ((size_t)split_blocks(a, K) * 4 + 255) / 256 * 256; }
size_t split_bytes(const DenseArgs &a, int64_t K)
{
    return presplit(a) ? odd_bytes(a, K) + (size_t)a.n_tiles * (size_t)((K + BK - 1) / BK) * 3 * (size_t)a.bn * 64 : 0;
}

template <bool KC_A, bool KC_B>
cudaError_t launch_dense(const DenseArgs &a, unsigned grid, bool pre, cudaStream_t st)
{
    if (!pre) {
        auto kern = dense_kernel<KC_A, KC_B, false>;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             Raw<KC_A, KC_B, false>::SMEM);
        if (e != cudaSuccess)
            return e;
        kern<<<grid, THREADS, Raw<KC_A, KC_B, false>::SMEM, st>>>(a);
        return cudaGetLastError();
    }
    auto kern = dense_kernel<KC_A, KC_B, true>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         Raw<KC_A, KC_B, true>::SMEM);
    if (e != cudaSuccess)
        return e;
    split_weights_kernel<KC_B><<<(unsigned)a.odd_words, 256, 0, st>>>(a, const_cast<unsigned char *>(a.Bs));
    e = cudaGetLastError();
    return e != cudaSuccess ? e : launch_dependent(kern, dim3(grid), THREADS, Raw<KC_A, KC_B, true>::SMEM, st, a);
}

}  // namespace

extern "C" int pspmm_dense_scratch_bytes(int64_t M, int64_t N, int64_t K, size_t *bytes)
{
    if (M < 0 || N < 0 || K < 0 || !bytes)
        return PSPMM_E_ARG;
    *bytes = 0;
    if (M == 0 || N == 0 || K == 0)
        return PSPMM_OK;
    DenseArgs a;
    plan(M, N, K, a);
    *bytes = partial_bytes(a, M, N) + split_bytes(a, K);
    return PSPMM_OK;
}

static int dense_run(int32_t transA, int32_t transB, int64_t M, int64_t N, int64_t K, const float *A, int64_t ldA,
                     const float *B, int64_t ldB, float *C, int64_t ldC, void *scratch, size_t scratch_bytes,
                     uint32_t wait_ns, int32_t withhold, void *stream)
{
    if (M < 0 || N < 0 || K < 0 || ldC < N || ldA < (transA ? M : K) || ldB < (transB ? K : N))
        return PSPMM_E_ARG;
    if (M == 0 || N == 0)
        return PSPMM_OK;
    if (!C || (K > 0 && (!A || !B)))
        return PSPMM_E_ARG;
    if (M > INT32_MAX - 1024 || K > INT32_MAX - 1024 || N > (1 << 20))
        return PSPMM_E_RANGE;
    cudaStream_t st = (cudaStream_t)stream;
    if (K == 0) {
        PSPMM_CUDA_TRY(cudaMemset2DAsync(C, (size_t)ldC * 4, 0, (size_t)N * 4, (size_t)M, st));
        return PSPMM_OK;
    }
    DenseArgs a;
    plan(M, N, K, a);
    a.A = A;
    a.B = B;
    a.ldA = ldA;
    a.ldB = ldB;
    a.M = (int32_t)M;
    a.N = (int32_t)N;
    a.K = (int32_t)K;
    a.C = C;
    a.ldC = ldC;
    a.wait_ns = wait_ns;
    a.withhold = withhold;
    const size_t need = partial_bytes(a, M, N) + split_bytes(a, K);
    if (need > 0 && (!scratch || scratch_bytes < need || (uintptr_t)scratch % 16 != 0))
        return PSPMM_E_ARG;
    if (a.splits > 1) {
        a.C = (float *)scratch;
        a.ldC = N;
    }
    const bool pre = presplit(a);
    a.odd = (unsigned *)((char *)scratch + partial_bytes(a, M, N));
    a.odd_words = (int32_t)split_blocks(a, K);
    a.Bs = (const unsigned char *)a.odd + odd_bytes(a, K);
    a.vecA = ldA % 4 == 0 && (uintptr_t)A % 16 == 0;
    a.vecB = ldB % 4 == 0 && (uintptr_t)B % 16 == 0;
    const int64_t items = (int64_t)a.m_tiles * a.n_tiles * a.splits;
    if (items > INT32_MAX - 65536)
        return PSPMM_E_RANGE;
    const unsigned grid = (unsigned)(items < pspmm_sm_count() ? items : pspmm_sm_count());
    // A is k-contiguous unless it is read transposed; B's rows are the output's columns.
    cudaError_t e;
    if (transA)
        e = transB ? launch_dense<false, true>(a, grid, pre, st) : launch_dense<false, false>(a, grid, pre, st);
    else
        e = transB ? launch_dense<true, true>(a, grid, pre, st) : launch_dense<true, false>(a, grid, pre, st);
    PSPMM_CUDA_TRY(e);
    if (a.splits > 1) {
        const ReduceArgs r = {a.C, C, ldC, a.splits, a.M, a.N};
        PSPMM_CUDA_TRY(launch_dependent(reduce_splits_kernel, dim3((unsigned)((M * N + 31) / 32)), 256, 0, st, r));
    }
    return PSPMM_OK;
}

extern "C" int pspmm_dense_mm(int32_t transA, int32_t transB, int64_t M, int64_t N, int64_t K, const float *A, int64_t ldA,
                              const float *B, int64_t ldB, float *C, int64_t ldC, void *scratch, size_t scratch_bytes,
                              void *stream)
{
    return dense_run(transA, transB, M, N, K, A, ldA, B, ldB, C, ldC, scratch, scratch_bytes, 2000000000u, 0, stream);
}

extern "C" int pspmm_dense_mm_stalled(int32_t transA, int32_t transB, int64_t M, int64_t N, int64_t K, const float *A,
                                      int64_t ldA, const float *B, int64_t ldB, float *C, int64_t ldC, void *scratch,
                                      size_t scratch_bytes, void *stream)
{
    return dense_run(transA, transB, M, N, K, A, ldA, B, ldB, C, ldC, scratch, scratch_bytes, 20000000u, 1, stream);
}

extern "C" int pspmm_dense_status(int32_t *status)
{
    if (!status)
        return PSPMM_E_ARG;
    unsigned v = 0;
    PSPMM_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_dense_status, sizeof(v)));
    *status = (int32_t)v;
    return PSPMM_OK;
}
