// Exact inner-product search with the tensor cores as a filter (dimensions up to 128).
//
// Same result as exact_topk_kernel: the k smallest (-<q,x>, id), the dot product accumulated in fp32 in d order without
// fused multiply-add.  Two fp32 operations per pair and dimension bound that kernel; here every pair costs a tensor
// product in fp16 and only a few hundred candidates per query are computed exactly:
//   * base and queries are scaled by powers of two (the base by tiles of 256 vectors, every query by itself) so that no
//     coordinate exceeds 1 and rounded to fp16; the sweep brings the products of a tile to the scale of the whole base;
//   * a sweep over all pairs keeps, per query, the largest product of every group of 32 base vectors;
//     (the last group, when the base ends inside it, is computed exactly in any case)
//   * with A the k-th largest of a query's group maxima and m a bound on the error of a product, k vectors have an exact
//     dot product of at least A - m, so only groups whose maximum reaches A - 2 m can hold one of the k best.  Their
//     vectors are computed exactly, those that reach A - m are sorted, the k first are the result.
// The bound: rounding both operands costs at most 2^-10 |q||x| plus 2^-25 per coordinate (the spacing of the smallest
// fp16 numbers), the sums of either side less than 2^-14 |q||x| at 128 terms; |x| is the largest norm of the base.
// A query whose candidates do not fit the buffers (products that hardly differ), a base or query with a number that is
// not finite: those queries are flagged and go to exact_topk_kernel, whose blocks otherwise end at once.
//
// The sweep has the shape of knn_mma.cu: 256 queries resident in shared memory (64 KB), base tiles of 256 in two stages,
// accumulators of 128 x 256 fp32 in the two halves of tensor memory, epilogue warps that take the tiles in turn.
#include <cuda_fp16.h>

#include "mma_common.cuh"

namespace cpb {
namespace {

using knn::kFull;
using knn::kWaitLimit;
using knn::mbar_wait_bounded;
using knn::smem_u32;
using namespace mma;

constexpr int kXmEpiWarps = 16;
constexpr int kXmThreads = (kXmEpiWarps + 2) * 32;
constexpr uint32_t kXmGroup = 32;          // base vectors per maximum
constexpr uint32_t kPickGroups = 1024;     // groups a query may list
constexpr uint32_t kPickKeys = 1024;       // candidates a query may sort
constexpr int kPickThreads = 256;

// A power of two that brings the largest coordinate, given by its bits, to at most 1; 0: not to be searched here.
__device__ __forceinline__ float scale_of(uint32_t big) {
    const int e = int(big >> 23);
    if (big == 0) return 1.0f;
    return e >= 64 && e <= 190 ? __uint_as_float(uint32_t(253 - e) << 23) : 0.0f;
}
// the base's scale, from its largest coordinate in stat[0]
__device__ __forceinline__ float base_scale(const uint32_t* stat) { return scale_of(stat[0]); }
// A tile's scale: 2^62, that of the smallest base that is searched, where all its coordinates are smaller still or zero (they
// stay below 1/2, and products at 2^62 are brought to the base's scale, 2^62 or less, like any others').
__device__ __forceinline__ float tile_scale_of(uint32_t big) { return scale_of(max(big, 64u << 23)); }

// ---- norms and largest coordinates: one warp per row -------------------------------------------------------------------
// per_row: {scale, scaled norm} of every query.
__global__ void row_stats_kernel(const float* __restrict__ x, uint64_t n, int dim, float2* __restrict__ per_row) {
    const int lane = threadIdx.x & 31;
    const uint64_t warps = uint64_t(gridDim.x) * (blockDim.x >> 5);
    const bool vec4 = (dim & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;  // (dim <= 128: a load per lane)
#pragma unroll 4
    for (uint64_t row = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; row < n; row += warps) {
        float sum = 0.0f;
        uint32_t big = 0;
        if (vec4) {
            if (4 * lane < dim) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(x + row * dim) + lane);
                big = max(max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu),
                          max(__float_as_uint(v.z) & 0x7fffffffu, __float_as_uint(v.w) & 0x7fffffffu));
                sum = v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
            }
        } else {
            for (int i = lane; i < dim; i += 32) {
                const float v = __ldg(x + row * dim + i);
                big = max(big, __float_as_uint(v) & 0x7fffffffu);
                sum += v * v;
            }
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
        big = __reduce_max_sync(kFull, big);
        const float len = sqrtf(sum) * 1.0001f;
        if (lane == 0) {
            const float scale = scale_of(big);
            per_row[row] = make_float2(scale, len * scale);
        }
    }
}

// ---- operand: [tile of 256 rows][chunk][row][8 halves] ------------------------------------------------------------------
__global__ void to_half_kernel(const float* __restrict__ x, uint64_t n, int dim, int chunks, const float2* __restrict__ per_row,
                               uint4* __restrict__ out, uint64_t tiles) {
    const uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t row = t / chunks;
    const int c = int(t % chunks);
    if (row >= tiles * kMmaRows) return;
    uint4 w = make_uint4(0u, 0u, 0u, 0u);
    if (row < n) {
        const float s = per_row[row].x;
        __half2 h[4];
        const float* src = x + row * dim + c * 8;
        if ((dim & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 a = c * 8 < dim ? __ldg(reinterpret_cast<const float4*>(src)) : zero;
            const float4 b = c * 8 + 4 < dim ? __ldg(reinterpret_cast<const float4*>(src) + 1) : zero;
            h[0] = __floats2half2_rn(a.x * s, a.y * s);
            h[1] = __floats2half2_rn(a.z * s, a.w * s);
            h[2] = __floats2half2_rn(b.x * s, b.y * s);
            h[3] = __floats2half2_rn(b.z * s, b.w * s);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float a = c * 8 + 2 * i < dim ? __ldg(src + 2 * i) : 0.0f, b = c * 8 + 2 * i + 1 < dim ? __ldg(src + 2 * i + 1) : 0.0f;
                h[i] = __floats2half2_rn(a * s, b * s);
            }
        }
        w = make_uint4(*reinterpret_cast<uint32_t*>(&h[0]), *reinterpret_cast<uint32_t*>(&h[1]), *reinterpret_cast<uint32_t*>(&h[2]),
                       *reinterpret_cast<uint32_t*>(&h[3]));
    }
    out[(row / kMmaRows * chunks + c) * kMmaRows + row % kMmaRows] = w;
}

// A tile of the base in one pass: its vectors in registers, 16 to a warp and four coordinates to a lane, their largest
// coordinate and norm, then the halves at the tile's own scale, chunk by chunk through shared memory (a chunk's rows 16
// bytes further apart in the banks than 4 KB) as contiguous copies.  What bounds it is the base's bytes: 500k x 128 are read
// once, 77 us (5.0 TB/s); with a pass for the statistics before the conversion 121.
// stat[0]: bits of the base's largest |coordinate|, stat[1]: bits of its largest norm (both non-negative floats, which order
// as integers; a number that is not finite shows as 0x7f800000 and above).
constexpr int kTileWarps = 16, kTileRows = kMmaRows / kTileWarps;
constexpr uint32_t kChunkStride = kMmaRows * 16 + 16;
__global__ void __launch_bounds__(kTileWarps * 32) base_tile_kernel(const float* __restrict__ x, uint64_t n, int dim, int chunks,
                                                                    uint32_t* __restrict__ stat, float* __restrict__ tile_scale,
                                                                    unsigned char* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char tile_smem[];
    __shared__ uint32_t top, longest;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t row0 = uint64_t(blockIdx.x) * kMmaRows + warp * kTileRows;
    const bool vec4 = (dim & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    if (threadIdx.x == 0) top = longest = 0;
    __syncthreads();
    float4 v[kTileRows];
#pragma unroll
    for (int i = 0; i < kTileRows; ++i) {
        v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row0 + i < n) {
            const float* src = x + (row0 + i) * dim + 4 * lane;
            if (vec4) {
                if (4 * lane < dim) v[i] = __ldg(reinterpret_cast<const float4*>(src));
            } else {
                if (4 * lane < dim) v[i].x = __ldg(src);
                if (4 * lane + 1 < dim) v[i].y = __ldg(src + 1);
                if (4 * lane + 2 < dim) v[i].z = __ldg(src + 2);
                if (4 * lane + 3 < dim) v[i].w = __ldg(src + 3);
            }
        }
    }
    uint32_t big = 0;
    float most = 0.0f;  // of the squared norms
    bool odd = false;   // one of them is not a number
#pragma unroll
    for (int i = 0; i < kTileRows; ++i) {
        big = max(big, max(max(__float_as_uint(v[i].x) & 0x7fffffffu, __float_as_uint(v[i].y) & 0x7fffffffu),
                           max(__float_as_uint(v[i].z) & 0x7fffffffu, __float_as_uint(v[i].w) & 0x7fffffffu)));
        float sum = v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
        odd = odd || !(sum >= 0.0f);
        most = fmaxf(most, sum);
    }
    big = __reduce_max_sync(kFull, big);
    if (lane == 0) {
        atomicMax(&top, big);
        atomicMax(&longest, odd ? 0x7fffffffu : __float_as_uint(sqrtf(most) * 1.0001f));
    }
    __syncthreads();
    // (a tile whose coordinates are too large has scale 0 and keeps the whole base from being searched here, by stat)
    const float s = tile_scale_of(top);
    if (threadIdx.x == 0) {
        atomicMax(stat, top);
        atomicMax(stat + 1, longest);
        tile_scale[blockIdx.x] = s;
    }
    if (lane < chunks * 2) {
#pragma unroll
        for (int i = 0; i < kTileRows; ++i) {
            const __half2 a = __floats2half2_rn(v[i].x * s, v[i].y * s), b = __floats2half2_rn(v[i].z * s, v[i].w * s);
            *reinterpret_cast<uint2*>(tile_smem + (lane >> 1) * kChunkStride + (warp * kTileRows + i) * 16 + (lane & 1) * 8) =
                make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
        }
    }
    __syncthreads();
    uint4* dst = reinterpret_cast<uint4*>(out + size_t(blockIdx.x) * chunks * kMmaRows * 16);
    for (int i = threadIdx.x; i < chunks * kMmaRows; i += kTileWarps * 32)
        dst[i] = *reinterpret_cast<const uint4*>(tile_smem + (i / kMmaRows) * kChunkStride + (i % kMmaRows) * 16);
}

// ---- sweep ----------------------------------------------------------------------------------------------------------------
// D fp32, A and B fp16, both K-major, M = 128, N = 256
constexpr uint32_t kXmIdesc = (1u << 4) | (uint32_t(256 >> 3) << 17) | (uint32_t(128 >> 4) << 24);

__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(kXmIdesc), "r"(uint32_t(accumulate))
        : "memory");
}
// 16 columns of the warp's 32 lanes of tensor memory: asked for, and waited for
__device__ __forceinline__ void tmem_load16f(float (&r)[16], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]),
          "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
        : "r"(addr)
        : "memory");
}
// (the registers are operands so that no use of them moves in front of the wait)
__device__ __forceinline__ void tmem_waitf(float (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]), "+f"(r[8]),
                   "+f"(r[9]), "+f"(r[10]), "+f"(r[11]), "+f"(r[12]), "+f"(r[13]), "+f"(r[14]), "+f"(r[15])
                 :
                 : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max16(const float (&r)[16]) {
    const float a = max3(r[0], r[1], r[2]), b = max3(r[3], r[4], r[5]), c = max3(r[6], r[7], r[8]), d = max3(r[9], r[10], r[11]);
    return max3(max3(a, b, c), max3(d, r[12], r[13]), fmaxf(r[14], r[15]));
}

struct SweepArgs {
    const uint4* queries;  // [tiles of 256 queries][chunks][256]
    const uint4* base;     // [tiles][chunks][256]
    const float* tile_scale;
    const uint32_t* stat;
    int chunks;
    uint64_t n;
    uint32_t nq, groups;   // groups: maxima per query (8 per tile)
    Split split;
    float* maxima;         // [nq][groups]
    uint32_t* status;      // this call's own: a lost wait sends the queries to exact_topk_kernel, no result is invalid
    uint32_t first_wait_polls;
};

__global__ void __launch_bounds__(kXmThreads, 1) exact_sweep_kernel(SweepArgs a) {
    extern __shared__ __align__(1024) unsigned char xm_smem[];
    __shared__ __align__(8) uint64_t full_bar[2], empty_bar[2], tfull_bar[2][2], tempty_bar[2][2], drain_bar;
    __shared__ uint32_t tmem_base_sm;
    __shared__ int abort_flag;
    const int lane = threadIdx.x & 31, warp = __shfl_sync(kFull, int(threadIdx.x >> 5), 0);
    const uint32_t operand_bytes = uint32_t(a.chunks) * kMmaRows * 16;
    constexpr uint32_t kStepBytes = 2 * kMmaRows * 16;
    const int ksteps = a.chunks / 2;  // 16 values of K a step: two 16-byte chunks
    unsigned char* a_sm = xm_smem;
    unsigned char* b_sm = xm_smem + operand_bytes;
    const uint64_t s0 = a.split.first_step(blockIdx.x);
    const uint32_t steps = uint32_t(a.split.first_step(blockIdx.x + 1) - s0);
    const uint32_t rt0 = uint32_t(s0 / a.split.cts), ct0 = uint32_t(s0 % a.split.cts);
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            knn::mbar_init(&full_bar[i], 1);
            knn::mbar_init(&empty_bar[i], 1);
            for (int j = 0; j < 2; ++j) {
                knn::mbar_init(&tfull_bar[i][j], 1);
                knn::mbar_init(&tempty_bar[i][j], 4);
            }
        }
        knn::mbar_init(&drain_bar, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kXmEpiWarps + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sm)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_sm;
    volatile int* aborted = &abort_flag;

    uint32_t loads = 0;
    if (warp == kXmEpiWarps) {
        if (lane == 0) {
            uint32_t rt = rt0, ct = ct0;
            bool fresh = true, ok = true;  // fresh: another tile of queries
            for (uint32_t i = 0; i < steps && ok && !*aborted; ++i) {
                const uint32_t s = i & 1;
                ok = wait_or_abort(&empty_bar[s], ((i >> 1) & 1) ^ 1, kWaitLimit, aborted);
                // it replaces the one that the step before still reads
                if (ok && fresh && i) ok = wait_or_abort(&empty_bar[s ^ 1], ((i - 1) >> 1) & 1, kWaitLimit, aborted);
                if (!ok) break;
                knn::mbar_expect_tx(&full_bar[s], fresh ? 2 * operand_bytes : operand_bytes);
                if (fresh) knn::bulk_g2s(a_sm, reinterpret_cast<const unsigned char*>(a.queries) + size_t(rt) * operand_bytes, operand_bytes, &full_bar[s]);
                knn::bulk_g2s(b_sm + s * operand_bytes, reinterpret_cast<const unsigned char*>(a.base) + size_t(ct) * operand_bytes, operand_bytes,
                              &full_bar[s]);
                ++loads;
                fresh = ++ct == a.split.cts;
                if (fresh) ct = 0, ++rt;
            }
            if (!ok) *aborted = 1;
        }
    } else if (warp == kXmEpiWarps + 1) {
        // the whole warp goes along and one lane issues: descriptors then stay in uniform registers
        const uint32_t elected = elect_one();
        const uint64_t a_desc = operand_desc(smem_u32(a_sm));
        const uint64_t b_desc[2] = {operand_desc(smem_u32(b_sm)), operand_desc(smem_u32(b_sm + operand_bytes))};
        bool ok = true;
        for (uint32_t i = 0; i < steps && ok; ++i) {
            const uint32_t s = i & 1;
            ok = __all_sync(kFull, wait_or_abort(&full_bar[s], (i >> 1) & 1, i == 0 ? a.first_wait_polls : kWaitLimit, aborted) && !*aborted);
            for (int h = 0; h < 2 && ok; ++h) {
                if (i) ok = __all_sync(kFull, wait_or_abort(&tempty_bar[h][s ^ 1], ((i - 1) >> 1) & 1, kWaitLimit, aborted));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint64_t ad = a_desc + h * ((128 * 16) >> 4), bd = b_desc[s];
                if (elected) {
#pragma unroll 4
                    for (int ks = 0; ks < ksteps; ++ks, ad += kStepBytes >> 4, bd += kStepBytes >> 4) mma_f16(tmem + h * 256, ad, bd, ks != 0);
                    mma_commit(&tfull_bar[h][s]);
                    if (h == 1) mma_commit(&empty_bar[s]);
                }
            }
        }
        if (!ok) *aborted = 1;
        if (elected) mma_commit(&drain_bar);  // everything issued above has finished when this completes
    } else {
        const int quarter = warp & 3, half = (warp >> 2) & 1, side = warp >> 3;
        const uint32_t local = uint32_t(half * 128 + quarter * 32 + lane), n = uint32_t(a.n);
        const uint32_t addr = tmem + (uint32_t(quarter * 32) << 16) + half * 256;
        const float whole = base_scale(a.stat);
        bool ok = true;
        for (uint32_t i = side; i < steps; i += 2) {
            const uint64_t step = s0 + i;
            const uint32_t q = uint32_t(step / a.split.cts) * kMmaRows + local, ct = uint32_t(step % a.split.cts);
            const float tile = __ldg(a.tile_scale + ct), to_whole = tile > 0.0f ? whole / tile : 0.0f;  // (powers of two)
            ok = wait_or_abort(&tfull_bar[half][side], (i >> 1) & 1, kWaitLimit, aborted);
            if (__ballot_sync(kFull, !ok || *aborted)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float out[8], r0[16], r1[16];
            tmem_load16f(r0, addr);
#pragma unroll
            for (int g = 0; g < 8; ++g) {
                tmem_waitf(r0);
                tmem_load16f(r1, addr + g * 32 + 16);
                float m = max16(r0);
                tmem_waitf(r1);
                if (g < 7) tmem_load16f(r0, addr + g * 32 + 32);
                out[g] = fmaxf(m, max16(r1)) * to_whole;
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty_bar[half][side]);
            if (ct * kMmaRows + kMmaRows > n) {  // groups with columns past the last vector (whose products are 0)
#pragma unroll
                for (int g = 0; g < 8; ++g)
                    if (ct * kMmaRows + g * 32 + 32 > n) out[g] = -INFINITY;
            }
            if (q < a.nq) {
                float4* dst = reinterpret_cast<float4*>(a.maxima + size_t(q) * a.groups + size_t(ct) * 8);
                dst[0] = make_float4(out[0], out[1], out[2], out[3]);
                dst[1] = make_float4(out[4], out[5], out[6], out[7]);
            }
        }
        if (!ok) *aborted = 1;
    }
    __syncthreads();
    // copies and products in flight after a lost wait end before the block's memory goes away
    if (warp == kXmEpiWarps && lane == 0 && *aborted) {
        atomicExch(a.status, kStatusWaitTimeout);
        for (uint32_t i = loads > 2 ? loads - 2 : 0; i < loads; ++i) mbar_wait_bounded(&full_bar[i & 1], (i >> 1) & 1, kWaitLimit);
    }
    if (warp == kXmEpiWarps + 1) {
        if (lane == 0) mbar_wait_bounded(&drain_bar, 0, kWaitLimit);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
    __syncthreads();
}

// ---- exact distances of the groups that can hold one of the k best, and the result: one block per query -------------------
struct PickArgs {
    const float* maxima;   // [nq][groups]
    const float* base;
    const float* queries;
    const uint32_t* stat;
    const float2* per_query;
    const uint32_t* status;
    uint64_t n;
    uint32_t groups, k;
    int dim, vec4, vec8;
    uint32_t* ids;
    float* dist;
    uint8_t* flags;        // 1: left to exact_topk_kernel
};

// float -> uint32 with the same order
__device__ __forceinline__ uint32_t order_of(float v) {
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float value_of(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); }

// 32 bytes, 32-byte aligned, by one instruction
__device__ __forceinline__ void load_sector(float* v, const float* p) {
    asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}

__global__ void __launch_bounds__(kPickThreads) exact_pick_kernel(PickArgs a) {
    __shared__ uint64_t keys[kPickKeys];
    __shared__ float list_max[kPickGroups], tops[kPickThreads];
    __shared__ uint32_t list[kPickGroups];
    __shared__ __align__(16) float qv[128];
    __shared__ uint32_t n_list, n_keys;
    __shared__ float kth;
    const uint32_t tid = threadIdx.x, q = blockIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const float* mx = a.maxima + size_t(q) * a.groups;
    const float2 pq = a.per_query[q];
    const float sx = base_scale(a.stat);
    if (sx == 0.0f || pq.x == 0.0f || *a.status != kStatusOk || __uint_as_float(a.stat[1]) * sx > 1e6f) {
        if (tid == 0) a.flags[q] = 1;
        return;
    }
    for (int i = tid; i < 128; i += kPickThreads) qv[i] = i < a.dim ? __ldg(a.queries + size_t(q) * a.dim + i) : 0.0f;
    if (tid == 0) n_list = 0, n_keys = 0;
    const float X = __uint_as_float(a.stat[1]) * sx;
    const float m = pq.y * X * (1.0f / 1024 + 1.0f / 8192) + sqrtf(float(a.dim)) * (pq.y + X) * (1.0f / 16777216);
    // The k-th largest of the threads' own maxima (256 of them, k <= 128) bounds A from below: A is found among the few
    // maxima that reach it, and what reaches A - 2 m is listed.  (A radix selection over all maxima spent its time in
    // atomics on few bins.)
    const float4* mx4 = reinterpret_cast<const float4*>(mx);
    float top = -INFINITY;
#pragma unroll 4
    for (uint32_t g = tid; g < a.groups / 4; g += kPickThreads) {
        const float4 v = __ldg(mx4 + g);
        top = fmaxf(fmaxf(top, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
    }
    tops[tid] = top;
    __syncthreads();
    {
        uint32_t above = 0;
#pragma unroll 8
        for (uint32_t i = 0; i < kPickThreads; ++i) above += tops[i] > top || (tops[i] == top && i < tid);
        if (above == a.k - 1) kth = top;
    }
    __syncthreads();
    // (the ragged group, whose maximum is -inf, joins the second list)
    const uint32_t ragged = a.n % kXmGroup ? uint32_t(a.n / kXmGroup) : kFull;
    float low = kth;
    for (int round = 0; round < 2; ++round) {
#pragma unroll 4
        for (uint32_t g4 = tid; g4 < a.groups / 4; g4 += kPickThreads) {
            const float4 v = __ldg(mx4 + g4);
            const float w[4] = {v.x, v.y, v.z, v.w};
            if (fmaxf(fmaxf(w[0], w[1]), fmaxf(w[2], w[3])) >= low || (round == 1 && g4 == ragged / 4)) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (w[i] >= low || (round == 1 && g4 * 4 + i == ragged)) {
                        const uint32_t at = atomicAdd(&n_list, 1u);
                        if (at < kPickGroups) {
                            list[at] = g4 * 4 + i;
                            list_max[at] = w[i];
                        }
                    }
            }
        }
        __syncthreads();
        const uint32_t listed = n_list;
        if (listed > kPickGroups || !(low > -INFINITY)) {
            if (tid == 0) a.flags[q] = 1;
            return;
        }
        if (round == 0) {  // A: the k-th of them
            for (uint32_t e = tid; e < listed; e += kPickThreads) {
                const float v = list_max[e];
                uint32_t above = 0;
#pragma unroll 8
                for (uint32_t i = 0; i < listed; ++i) above += list_max[i] > v || (list_max[i] == v && i < e);
                if (above == a.k - 1) kth = v;
            }
            __syncthreads();
            low = kth - 2.0f * m;
            if (tid == 0) n_list = 0;
            __syncthreads();
        }
    }
    const uint32_t groups = n_list;
    const float fine = kth - m;
    const float s = sx * pq.x;
    for (uint32_t i = warp; i < groups; i += kPickThreads / 32) {
        const uint64_t id = uint64_t(list[i]) * kXmGroup + lane;
        if (id < a.n) {
            const float* x = a.base + id * a.dim;
            float dot = 0.0f;
            if (a.vec8) {  // whole sectors: half the requests of 16-byte loads, whose second halves mostly missed L1 again
#pragma unroll 1
                for (int d0 = 0; d0 < a.dim; d0 += 16) {
                    float v[16];
                    load_sector(v, x + d0);
                    if (d0 + 8 < a.dim) load_sector(v + 8, x + d0 + 8);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float4 u = *reinterpret_cast<const float4*>(qv + d0 + 4 * c);
                        if (c < 2 || d0 + 8 < a.dim) {
                            dot = __fadd_rn(dot, __fmul_rn(u.x, v[4 * c]));
                            dot = __fadd_rn(dot, __fmul_rn(u.y, v[4 * c + 1]));
                            dot = __fadd_rn(dot, __fmul_rn(u.z, v[4 * c + 2]));
                            dot = __fadd_rn(dot, __fmul_rn(u.w, v[4 * c + 3]));
                        }
                    }
                }
            } else if (a.vec4) {
// a lane reads 64 bytes of its vector at once: a sector's two halves are then asked for together
#pragma unroll 1
                for (int d0 = 0; d0 < a.dim; d0 += 16) {
                    float4 v[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) v[c] = d0 + 4 * c < a.dim ? __ldg(reinterpret_cast<const float4*>(x + d0) + c) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float4 u = *reinterpret_cast<const float4*>(qv + d0 + 4 * c);  // (zeros past the last dimension)
                        if (d0 + 4 * c < a.dim) {
                            dot = __fadd_rn(dot, __fmul_rn(u.x, v[c].x));
                            dot = __fadd_rn(dot, __fmul_rn(u.y, v[c].y));
                            dot = __fadd_rn(dot, __fmul_rn(u.z, v[c].z));
                            dot = __fadd_rn(dot, __fmul_rn(u.w, v[c].w));
                        }
                    }
                }
            } else {
                for (int d = 0; d < a.dim; ++d) dot = __fadd_rn(dot, __fmul_rn(qv[d], __ldg(x + d)));
            }
            if (!(dot * s < fine)) {
                const uint32_t at = atomicAdd(&n_keys, 1u);
                // 0 - dot: the negated dot product with one zero (+0) only
                if (at < kPickKeys) keys[at] = uint64_t(order_of(__fsub_rn(0.0f, dot))) << 32 | uint32_t(id);
            }
        }
    }
    __syncthreads();
    const uint32_t found = n_keys;
    if (found > kPickKeys || found < a.k) {
        if (tid == 0) a.flags[q] = 1;
        return;
    }
    for (uint32_t e = tid; e < found; e += kPickThreads) {  // rank by counting: keys are distinct
        const uint64_t key = keys[e];
        uint32_t rank = 0;
#pragma unroll 4
        for (uint32_t i = 0; i < found; ++i) rank += keys[i] < key;
        if (rank < a.k) {
            a.ids[size_t(q) * a.k + rank] = uint32_t(key);
            a.dist[size_t(q) * a.k + rank] = value_of(uint32_t(key >> 32));
        }
    }
    if (tid == 0) a.flags[q] = 0;
}

}  // namespace

// Needs several groups per result to bound the k-th best from; below 16,384 vectors the launches cost more than the plain
// kernel.  (4 queries on 20k / 300k x 128: 109 / 485 us on the plain kernel, 64 queries here: 75 / 167 us.)
bool exact_mma_supported(const cphnsw_b200_index* h, uint64_t n, uint64_t nq, uint32_t k) {
    return h->dim <= 128 && n >= 16384 && n < 0x80000000ull && n / kXmGroup >= 4ull * k && nq < 0x7fffffffull;
}

// Writes the results of all queries but the flagged ones; flags uint8[nq] (device).
int launch_exact_mma(cphnsw_b200_index* h, const float* d_base, uint64_t n, const float* d_q, uint64_t nq, uint32_t k, uint32_t* d_ids,
                     float* d_dist, uint8_t* d_flags, cudaStream_t st) {
    const int dim = int(h->dim), chunks = (dim + 15) / 16 * 2;
    const uint64_t tiles = (n + kMmaRows - 1) / kMmaRows, groups = tiles * (kMmaRows / kXmGroup);
    const size_t operand_bytes = size_t(chunks) * kMmaRows * 16;
    // queries go in batches whose maxima take at most 512 MB (whole tiles of queries, one at least)
    uint64_t batch = (size_t(512) << 20) / (groups * 4) / kMmaRows * kMmaRows;
    if (batch < kMmaRows) batch = kMmaRows;
    if (batch > nq) batch = nq;
    const uint64_t qtiles = (batch + kMmaRows - 1) / kMmaRows;
    auto up = [](size_t b) { return (b + 255) & ~size_t(255); };
    const size_t base_b = up(size_t(tiles) * operand_bytes), q_b = up(size_t(qtiles) * operand_bytes);
    const size_t max_b = up(size_t(batch) * groups * 4), row_b = up(size_t(batch) * 8), scale_b = up(size_t(tiles) * 4);
    CPB_TRY(reserve_workspace(h, h->s_exact, 256 + base_b + q_b + max_b + row_b + scale_b));
    unsigned char* p = h->s_exact.as<unsigned char>();
    uint32_t* stat = reinterpret_cast<uint32_t*>(p);
    uint4* base_op = reinterpret_cast<uint4*>(p + 256);
    uint4* q_op = reinterpret_cast<uint4*>(p + 256 + base_b);
    float* maxima = reinterpret_cast<float*>(p + 256 + base_b + q_b);
    float2* per_query = reinterpret_cast<float2*>(p + 256 + base_b + q_b + max_b);
    float* tile_scale = reinterpret_cast<float*>(p + 256 + base_b + q_b + max_b + row_b);

    uint32_t* status = stat + 2;
    CPB_CUDA(cudaMemsetAsync(stat, 0, 12, st));
    const unsigned stat_blocks = unsigned(h->sm_count) * 8;
    CPB_CUDA(allow_max_dynamic_smem(base_tile_kernel));
    base_tile_kernel<<<unsigned(tiles), kTileWarps * 32, chunks * kChunkStride, st>>>(d_base, n, dim, chunks, stat, tile_scale,
                                                                                     reinterpret_cast<unsigned char*>(base_op));
    h->launches++;
    CPB_CUDA(cudaGetLastError());
    CPB_CUDA(allow_max_dynamic_smem(exact_sweep_kernel));
    for (uint64_t q0 = 0; q0 < nq; q0 += batch) {
        const uint64_t m = nq - q0 < batch ? nq - q0 : batch;
        const uint64_t rts = (m + kMmaRows - 1) / kMmaRows;
        const float* qs = d_q + q0 * dim;
        row_stats_kernel<<<unsigned((m + 7) / 8 < stat_blocks ? (m + 7) / 8 : stat_blocks), 256, 0, st>>>(qs, m, dim, per_query);
        const uint64_t q_cells = rts * kMmaRows * chunks;
        to_half_kernel<<<unsigned((q_cells + 255) / 256), 256, 0, st>>>(qs, m, dim, chunks, per_query, q_op, rts);
        SweepArgs a;
        a.queries = q_op;
        a.base = base_op;
        a.tile_scale = tile_scale;
        a.stat = stat;
        a.chunks = chunks;
        a.n = n;
        a.nq = uint32_t(m);
        a.groups = uint32_t(groups);
        a.split.cts = uint32_t(tiles);
        a.split.steps = rts * tiles;
        a.split.blocks = uint32_t(a.split.steps < uint64_t(h->sm_count) ? a.split.steps : uint64_t(h->sm_count));
        a.maxima = maxima;
        a.status = status;
        a.first_wait_polls = h->first_wait_polls;
        exact_sweep_kernel<<<a.split.blocks, kXmThreads, 3 * operand_bytes, st>>>(a);
        PickArgs b;
        b.maxima = maxima;
        b.base = d_base;
        b.queries = qs;
        b.stat = stat;
        b.per_query = per_query;
        b.status = status;
        b.n = n;
        b.groups = uint32_t(groups);
        b.k = k;
        b.dim = dim;
        b.vec4 = (dim & 3) == 0 && (reinterpret_cast<uintptr_t>(d_base) & 15) == 0 ? 1 : 0;
        b.vec8 = (dim & 7) == 0 && (reinterpret_cast<uintptr_t>(d_base) & 31) == 0 ? 1 : 0;
        b.ids = d_ids + q0 * k;
        b.dist = d_dist + q0 * k;
        b.flags = d_flags + q0;
        exact_pick_kernel<<<unsigned(m), kPickThreads, 0, st>>>(b);
        h->launches += 4;
        CPB_CUDA(cudaGetLastError());
    }
    return 0;
}

}  // namespace cpb
