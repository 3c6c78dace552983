// Cross-polytope encode: Psi(x) = H D3 H D2 H D1 x for K rotations, fused with the signed
// argmax that produces one code component per rotation.
//
// What it computes follows the reference's RandomHadamardRotation::apply_copy
// (include/cphnsw/encoder/rotation.hpp:90-111), fht (include/cphnsw/encoder/transform/fht.hpp),
// detail::find_argmax_abs (include/cphnsw/encoder/cp_encoder.hpp:25-92) and CPCode::encode
// (include/cphnsw/core/types.hpp:88-90).  Bit-exactness rests on three facts:
//   * every butterfly is one IEEE add or subtract in the stage order h = 1, 2, 4, ... — the
//     kernels use __fadd_rn/__fsub_rn (never contracted) in that order;
//   * multiplying by a +-1 diagonal is exact, so folding it into the first butterfly stage as
//     fma(s1, x1, s0*x0) rounds exactly like (s0*x0) + (s1*x1);
//   * the reference's SIMD FHT differs from its scalar FHT only by negating element i when
//     popcount(i & (W-1)) is odd (W = 8 AVX2, 16 AVX-512).  The host folds that diagonal into
//     the sign tables of layers 1 and 2; the last one only decides the sign bit of the code
//     (and the sign of the rotated output), applied here through `flip_mask` = W-1.
//
// Five kernels:
//   encode_thread_kernel padded dims 32, 64 and 128 (d in 17..128): one thread owns one vector, the whole
//                        transform lives in registers (no shuffles, no barriers in the
//                        inner loop); the bound is the fp32 add pipe.
//   encode_warp_kernel   padded dims 256 and 512, few vectors: one warp per vector, P/32 consecutive elements per lane,
//                        low stages in registers, high stages by shuffles.
//   encode_group_kernel  padded dims 256 and 512, many vectors: 2 or 4 lanes own one vector, 128 elements each; the stages
//                        across lanes become register stages after an exchange.
//   encode_p1024_kernel  padded dim 1024: one warp per vector, register and lane bits change places through tensor memory.
//   encode_generic_kernel any other power-of-two padded dim: one warp owns one vector in shared memory.
#include "common.cuh"

namespace cpb {
namespace {

constexpr int kTileVecs = 128;          // vectors per block = threads per block
// Padded row of the staged tile: 64-bit reads of 16 threads hit distinct banks.  (Measured and dropped at
// P = 128: the diagonal applied as a sign-bit XOR on the integer pipe, which the argmax loads already, 3.81 ms per 1M
// vectors against 3.56 ms; the diagonal folded into every stage as block multipliers, 2 % slower.)
template <int P>
constexpr int kTileStride = P + 2;

// ---- packed fp32 pairs (two IEEE operations per instruction, each rounded as the scalar one) -----------------------
// The transform is bound by fp32 adds; packing leaves the add pipe as busy but halves the issue slots they take, which
// scalar code shared with the argmax and the table reads.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// butterflies between pairs H apart (elements 2 * H apart)
template <int H, int N>
__device__ __forceinline__ void butterfly_pairs(f32x2 (&v)[N]) {
#pragma unroll
    for (int i = 0; i < N; i += 2 * H) {
#pragma unroll
        for (int j = i; j < i + H; ++j) {
            const f32x2 x = v[j], y = v[j + H];
            v[j] = add2(x, y);
            v[j + H] = sub2(x, y);
        }
    }
}

template <int H, int N, int END = N>
__device__ __forceinline__ void butterfly_stages(f32x2 (&v)[N]) {
    if constexpr (H < END) {
        butterfly_pairs<H>(v);
        butterfly_stages<2 * H, N, END>(v);
    }
}

// D then H on P values held as pairs of neighbours.  `sg` points at P +-1 floats in shared memory, read by
// every thread at the same address (broadcast).  The products with +-1 are exact.
template <int P>
__device__ __forceinline__ void diag_fht(f32x2 (&v)[P / 2], const float* __restrict__ sg) {
    const ulonglong2* s2 = reinterpret_cast<const ulonglong2*>(sg);
#pragma unroll
    for (int c = 0; c < P / 4; ++c) {
        const ulonglong2 s = s2[c];
        float a, b;
        unpack2(mul2(v[2 * c], s.x), a, b);
        v[2 * c] = pack2(__fadd_rn(a, b), __fsub_rn(a, b));
        unpack2(mul2(v[2 * c + 1], s.y), a, b);
        v[2 * c + 1] = pack2(__fadd_rn(a, b), __fsub_rn(a, b));
    }
    butterfly_stages<1>(v);
}

// Lowest-index argmax of |v| by a left-biased tournament: the right operand wins only when it is
// strictly larger, so among equal magnitudes the lowest index survives every round
// (same answer as the strict `>` scan of cp_encoder.hpp:82-88).
template <int P>
__device__ __forceinline__ void argmax_abs(const f32x2 (&v)[P / 2], float& win, int& idx) {
    float w[P / 2];
    int id[P / 2];
#pragma unroll
    for (int j = 0; j < P / 2; ++j) {
        float a, b;
        unpack2(v[j], a, b);
        bool r = fabsf(b) > fabsf(a);
        w[j] = r ? b : a;
        id[j] = r ? 2 * j + 1 : 2 * j;
    }
#pragma unroll
    for (int n = P / 4; n >= 1; n >>= 1) {
#pragma unroll
        for (int j = 0; j < n; ++j) {
            bool r = fabsf(w[2 * j + 1]) > fabsf(w[2 * j]);
            w[j] = r ? w[2 * j + 1] : w[2 * j];
            id[j] = r ? id[2 * j + 1] : id[2 * j];
        }
    }
    win = w[0];
    idx = id[0];
}

// sign bit of the component: `value < 0` (cp_encoder.hpp:174) after the convention's last
// diagonal, which negates the value when popcount(idx & flip_mask) is odd.
__device__ __forceinline__ uint32_t component_of(float win, int idx, int flip_mask) {
    bool flip = __popc(idx & flip_mask) & 1;
    bool neg = flip ? (win > 0.0f) : (win < 0.0f);
    return (uint32_t(idx) << 1) | (neg ? 1u : 0u);
}

// The block's vectors, zero-padded, a thread's part of one (128 elements, or all of it) a row: coalesced 128-bit loads
// when rows are 16-byte aligned, else 32-bit loads, kStageRows rows in flight per warp (one at a time, the round trips of a
// warp's 32 rows in sequence took as long as a rotation: 10k x 128, K = 32, 58 us against 50, with rotated vectors 113 against
// 98; 2k x 256 47 against 37).
constexpr int kStageRows = 8;
template <int P>
__device__ __forceinline__ void stage_tile(float* tile, const float* __restrict__ x, uint64_t row0, int rows, int dim, int lane, int warp) {
    constexpr int W = P < 128 ? P : 128, G = P / W;  // elements of a row, rows per vector
    constexpr int kStride = kTileStride<W>, C = W / 32;
    const bool vec4 = (dim % 4 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
    for (int r0 = warp * kStageRows; r0 < kTileVecs; r0 += kTileVecs / 32 * kStageRows) {
        float4 q[kStageRows];
#pragma unroll
        for (int i = 0; i < kStageRows; ++i) {
            const int r = r0 + i, left = r / G < rows ? dim - W * (r % G) : 0;  // elements of the vector from this row on
            const float* src = x + (row0 + r / G) * uint64_t(dim) + W * (r % G);
            q[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (vec4) {
                if (4 * lane < left && 4 * lane < W) q[i] = __ldg(reinterpret_cast<const float4*>(src) + lane);
            } else {
                if (lane < left) q[i].x = __ldg(src + lane);
                if (C > 1 && lane + 32 < left) q[i].y = __ldg(src + lane + 32);
                if (C > 2 && lane + 64 < left) q[i].z = __ldg(src + lane + 64);
                if (C > 2 && lane + 96 < left) q[i].w = __ldg(src + lane + 96);
            }
        }
#pragma unroll
        for (int i = 0; i < kStageRows; ++i) {
            float* dst = tile + (r0 + i) * kStride;
            if (vec4) {
                if (4 * lane < W) {
                    f32x2* to = reinterpret_cast<f32x2*>(dst + 4 * lane);
                    to[0] = pack2(q[i].x, q[i].y);
                    to[1] = pack2(q[i].z, q[i].w);
                }
            } else {
                dst[lane] = q[i].x;
                if (C > 1) dst[lane + 32] = q[i].y;
                if (C > 2) dst[lane + 64] = q[i].z, dst[lane + 96] = q[i].w;
            }
        }
    }
}

// QUERY = true additionally writes the rotated vectors and winning magnitudes (CPQuery).  A vector a thread at padded
// dims 32 and 64 too: with a warp a vector the shuffles of the high stages (one an element) were the bound, 300k x 64 with
// K = 32 took 2.09 ms and takes 0.50, 300k x 32 took 1.64 and takes 0.24.  (Measured and dropped at P = 128: the second
// sign product in the fma of the first butterfly, 3.65 ms per 1M against 3.56.)
template <typename CompT, bool QUERY, int P>
__global__ void __launch_bounds__(kTileVecs, P == 128 ? (QUERY ? 2 : 3) : (P == 64 ? 5 : 8))
encode_thread_kernel(const float* __restrict__ x, uint64_t n, int dim, int K, int rpb /* rotations per block */,
                   const float* __restrict__ signs /*[K][3][P]*/, int flip_mask,
                   CompT* __restrict__ codes, float* __restrict__ rotated, float* __restrict__ mags) {
    extern __shared__ float smem[];
    float* tile = smem;                                                 // [kTileVecs][kTileStride<P>]
    float* sign_sm = tile + kTileVecs * kTileStride<P>;                              // [2][3][P], double buffer
    CompT* code_tile = reinterpret_cast<CompT*>(sign_sm + 2 * 3 * P);         // [kTileVecs][rotations of this block]
    const int r0 = blockIdx.y * rpb, r1 = min(K, r0 + rpb), nr = r1 - r0;

    const uint64_t row0 = uint64_t(blockIdx.x) * kTileVecs;
    const int rows = int(min(uint64_t(kTileVecs), n - row0));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    stage_tile<P>(tile, x, row0, rows, dim, lane, warp);
    // the three diagonals of one rotation are staged in shared memory one rotation ahead
    const int t = threadIdx.x;
    if (t < 3 * P / 4)
        reinterpret_cast<float4*>(sign_sm)[t] = __ldg(reinterpret_cast<const float4*>(signs + size_t(r0) * 3 * P) + t);
    __syncthreads();

    const f32x2* mine = reinterpret_cast<const f32x2*>(tile + t * kTileStride<P>);
    const uint64_t row = row0 + t;
    for (int r = r0; r < r1; ++r) {
        if (r + 1 < r1 && t < 3 * P / 4)
            reinterpret_cast<float4*>(sign_sm + ((r + 1 - r0) & 1) * 3 * P)[t] =
                __ldg(reinterpret_cast<const float4*>(signs + size_t(r + 1) * 3 * P) + t);
        f32x2 v[P / 2];
#pragma unroll
        for (int i = 0; i < P / 2; ++i) v[i] = mine[i];
        const float* sg = sign_sm + ((r - r0) & 1) * 3 * P;
#pragma unroll 1
        for (int layer = 0; layer < 3; ++layer) diag_fht<P>(v, sg + layer * P);
        float win;
        int idx;
        argmax_abs<P>(v, win, idx);
        code_tile[t * nr + (r - r0)] = CompT(component_of(win, idx, flip_mask));
        if (QUERY && t < rows) {
            if (mags) mags[row * K + r] = fabsf(win);
            if (rotated) {
                float* out = rotated + (row * K + r) * P;
                // (at 128 the code for both makes every small call 2 us longer, 10.7 us for 30 vectors against 8.8:
                // launch_encode sends other addresses elsewhere)
                const bool wide = P == 128 || (reinterpret_cast<uintptr_t>(rotated) & 15) == 0;
#pragma unroll
                for (int c = 0; c < P / 4; ++c) {
                    float a0, a1, a2, a3;
                    unpack2(v[2 * c], a0, a1);
                    unpack2(v[2 * c + 1], a2, a3);
                    float4 o;
                    o.x = (__popc((4 * c) & flip_mask) & 1) ? -a0 : a0;
                    o.y = (__popc((4 * c + 1) & flip_mask) & 1) ? -a1 : a1;
                    o.z = (__popc((4 * c + 2) & flip_mask) & 1) ? -a2 : a2;
                    o.w = (__popc((4 * c + 3) & flip_mask) & 1) ? -a3 : a3;
                    if (wide) reinterpret_cast<float4*>(out)[c] = o;
                    else out[4 * c] = o.x, out[4 * c + 1] = o.y, out[4 * c + 2] = o.z, out[4 * c + 3] = o.w;
                }
            }
        }
        __syncthreads();  // the next rotation's diagonals are in place, this rotation's are free
    }
    // the tile's codes are contiguous in the output (a row of K at a time when the rotations are split over blocks)
    CompT* dst = codes + row0 * uint64_t(K);
    if (nr == K) {
        for (int i = threadIdx.x; i < rows * K; i += kTileVecs) dst[i] = code_tile[i];
    } else {
        for (int i = threadIdx.x; i < rows * nr; i += kTileVecs) dst[uint64_t(i / nr) * K + r0 + i % nr] = code_tile[i];
    }
}

// ---- padded dim 1024 (d in 513..1024): one warp per vector, 32 elements per lane -------------------
// Five of an element's ten index bits are the register's, five the lane's, and a stage pairs registers, so bits have to
// change places as the stages go up.  They do by way of tensor memory: what a warp stores in one shape (16 lanes by 128 bits,
// eight such side by side, twice) it loads in another (32 lanes by 32 bits).  The lane that stores register r = R4 .. R0 (bits)
// with p4 .. p0 its own index puts it at lane R4 R0 p4 p3 p2 and column R3 R2 R1 p1 p0, and the one that loads has lane and
// column for lane and register: two of the lane's bits come to the registers, two of the registers' go to the lanes.
//   The vector starts with bits 0 1 8 5 2 as R0 .. R4 and 3 4 6 7 9 as p0 .. p4.  Stages 0, 1, 2 are those of R0, R1, R4; a
// change leaves bits 3 4 1 8 5 and 6 7 9 0 2, so the next three are again those of R0, R1, R4, and so on (all bits three up,
// modulo ten): 30 stages of three layers take nine changes.  Stage order and butterfly (lo = x + y, hi = x - y, x the lower
// index) are the reference's, so the result is bit-identical.  The diagonals come bit-packed in the order a layer finds the
// elements in (a set bit negates), one word per lane and layer.
//   What bounds it is the add pipe (0.61 of it) and the instructions beside: without the changes of places it would take 0.84 of
// its time, without two of the three diagonals 0.9, without the search for the argmax 0.93.  With transposes through shared
// memory, five of 64 wavefronts each a vector and rotation, these were the bound: 100k x 960, K = 32, 5,340 us; 4,390 now.
// Rotated vectors wanted, 2,000 of 960: 153 us with transposes, 118 now, although a lane then spills 10 to 18 registers.
//   Tensor memory is an SM's own: a block that finds all of it taken, by a kernel on another stream, stands until some is given
// back.  (Beside a block of the sweeps of this library, which take all, none has the registers to start.)
constexpr int kP1024 = 1024;
constexpr int kWarps1024 = 4;
constexpr int kBlocks1024 = 4;  // resident on an SM (five of 96 registers spill: 4,480 us)
constexpr uint32_t kTmemCols1024 = 32;

// the bit of an element's index that position `at` (R0 .. R4, p0 .. p4) holds after `changes` changes of places
__host__ __device__ constexpr int index_bit(int at, int changes) {
    const int first[10] = {0, 1, 8, 5, 2, 3, 4, 6, 7, 9};
    return (first[at] + 3 * changes) % 10;
}
__host__ __device__ constexpr int index_part(int value, int from, int changes) {  // of a register's number (from = 0), of a lane's (5)
    int i = 0;
    for (int b = 0; b < 5; ++b)
        if (value >> b & 1) i |= 1 << index_bit(from + b, changes);
    return i;
}

__device__ __forceinline__ void change_places(f32x2 (&p)[16], uint32_t tmem) {
    float v[32];
#pragma unroll
    for (int j = 0; j < 16; ++j) unpack2(p[j], v[2 * j], v[2 * j + 1]);
#pragma unroll
    for (int h = 0; h < 2; ++h)
        asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(
                         tmem + (uint32_t(h * 16) << 16)),
                     "f"(v[16 * h]), "f"(v[16 * h + 1]), "f"(v[16 * h + 2]), "f"(v[16 * h + 3]), "f"(v[16 * h + 4]), "f"(v[16 * h + 5]), "f"(v[16 * h + 6]),
                     "f"(v[16 * h + 7]), "f"(v[16 * h + 8]), "f"(v[16 * h + 9]), "f"(v[16 * h + 10]), "f"(v[16 * h + 11]), "f"(v[16 * h + 12]),
                     "f"(v[16 * h + 13]), "f"(v[16 * h + 14]), "f"(v[16 * h + 15])
                     : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, "
        "%21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]),
          "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]),
          "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
        : "r"(tmem)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) {  // (no use of them moves in front of the wait)
        asm volatile("" : "+f"(v[2 * j]), "+f"(v[2 * j + 1]));
        p[j] = pack2(v[2 * j], v[2 * j + 1]);
    }
}
// the stage of R0, the halves of a pair
__device__ __forceinline__ void butterfly_halves(f32x2 (&p)[16]) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        float a, b;
        unpack2(p[j], a, b);
        p[j] = pack2(__fadd_rn(a, b), __fsub_rn(a, b));
    }
}
__device__ __forceinline__ void flip_signs32(f32x2 (&p)[16], uint32_t word) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        float a, b;
        unpack2(p[j], a, b);
        a = __int_as_float(__float_as_int(a) ^ int((word << (31 - 2 * j)) & 0x80000000u));
        b = __int_as_float(__float_as_int(b) ^ int((word << (30 - 2 * j)) & 0x80000000u));
        p[j] = pack2(a, b);
    }
}

template <typename CompT, bool QUERY>
__global__ void __launch_bounds__(kWarps1024 * 32, kBlocks1024)
encode_p1024_kernel(const float* __restrict__ x, uint64_t n, int dim, int K, int rpb,
                    const uint32_t* __restrict__ signbits /*[K][3][32]*/, int flip_mask,
                    CompT* __restrict__ codes, float* __restrict__ rotated, float* __restrict__ mags) {
    __shared__ uint32_t tmem_base_sm;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(uint32_t(__cvta_generic_to_shared(&tmem_base_sm))),
                     "r"(kTmemCols1024)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_sm + (uint32_t(warp * 32) << 16);
    const bool vec4 = (dim % 4 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
    const int begins = index_part(lane, 5, 0);  // of the lane's elements, at first
    for (uint64_t row = uint64_t(blockIdx.x) * kWarps1024 + warp; row < n; row += uint64_t(gridDim.x) * kWarps1024) {
        // the vector, zero-padded; registers 4 c .. 4 c + 3 of a lane are neighbours (bits 0 and 1 of the index, and bits 8, 5, 2)
        f32x2 in[16];
        const float* src = x + row * uint64_t(dim);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int i = begins + index_part(4 * c, 0, 0);
            float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
            if (vec4) {
                if (i < dim) q = __ldg(reinterpret_cast<const float4*>(src + i));
            } else {
                if (i < dim) q.x = __ldg(src + i);
                if (i + 1 < dim) q.y = __ldg(src + i + 1);
                if (i + 2 < dim) q.z = __ldg(src + i + 2);
                if (i + 3 < dim) q.w = __ldg(src + i + 3);
            }
            in[2 * c] = pack2(q.x, q.y), in[2 * c + 1] = pack2(q.z, q.w);
        }
        for (int r = blockIdx.y * rpb; r < min(K, int(blockIdx.y + 1) * rpb); ++r) {
            const uint32_t* sb = signbits + size_t(r) * 3 * 32 + lane;
            const uint32_t word0 = __ldg(sb), word1 = __ldg(sb + 32), word2 = __ldg(sb + 64);
            f32x2 v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = in[j];
            flip_signs32(v, word0);
#pragma unroll
            for (int c = 0; c < 10; ++c) {  // stages 3 c, 3 c + 1, 3 c + 2 of 30; layers begin with the 10th and the 20th
                if (c) change_places(v, tmem);
                butterfly_halves(v);
                if (c == 3) flip_signs32(v, word1);
                butterfly_pairs<1>(v);
                if (c == 6) flip_signs32(v, word2);
                butterfly_pairs<8>(v);
            }
            // lowest-index argmax of |v|: the largest magnitude, then the first element that has it (from the last one down)
            float best = -1.0f, win = 0.0f;
            int idx = 0x7fffffff;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                float a, b;
                unpack2(v[j], a, b);
                best = fmaxf(best, fmaxf(fabsf(a), fabsf(b)));
            }
            best = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(best)));  // (none of them is above zero only where all are NaN)
#pragma unroll
            for (int e = 31; e >= 0; --e) {  // R3 R2 R0 R1 R4 hold bits 2 5 7 8 9
                const int reg = (e >> 2 & 3) | (e >> 1 & 1) << 2 | (e & 1) << 3 | (e >> 4) << 4;
                float a, b;
                unpack2(v[reg / 2], a, b);
                const float y = reg & 1 ? b : a;
                if (fabsf(y) == best) idx = index_part(reg, 0, 9), win = y;
            }
            if (idx != 0x7fffffff) idx += index_part(lane, 5, 9);
            const int least = __reduce_min_sync(0xffffffffu, idx);
            win = __shfl_sync(0xffffffffu, win, __ffs(__ballot_sync(0xffffffffu, idx == least)) - 1);
            if (lane == 0) {
                codes[row * K + r] = CompT(component_of(win, least, flip_mask));
                if (QUERY && mags) mags[row * K + r] = best;
            }
            if (QUERY && rotated) {
                change_places(v, tmem);  // back to where they began
                float* out = rotated + (row * K + r) * uint64_t(kP1024);
                const bool wide = (reinterpret_cast<uintptr_t>(rotated) & 15) == 0;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const int i = begins + index_part(4 * c, 0, 0);
                    float4 o;
                    unpack2(v[2 * c], o.x, o.y);
                    unpack2(v[2 * c + 1], o.z, o.w);
                    if (__popc(i & flip_mask) & 1) o.x = -o.x;
                    if (__popc((i + 1) & flip_mask) & 1) o.y = -o.y;
                    if (__popc((i + 2) & flip_mask) & 1) o.z = -o.z;
                    if (__popc((i + 3) & flip_mask) & 1) o.w = -o.w;
                    if (wide) *reinterpret_cast<float4*>(out + i) = o;
                    else out[i] = o.x, out[i + 1] = o.y, out[i + 2] = o.z, out[i + 3] = o.w;
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base_sm), "r"(kTmemCols1024) : "memory");
}

// ---- padded dims 256, 512: one warp per vector, E = P / 32 consecutive elements per lane ----------------------
// Lane L holds elements E*L .. E*L + E - 1.  Stages h < E pair elements of one lane (registers), stages
// h = E * 2^t pair lane L with lane L ^ 2^t (one shuffle per element): the lower index computes x + y, the upper
// x - y with x the lower element, in ascending h like the reference's loop (fht.hpp:56-69), so the result is
// bit-identical.  Nothing goes through shared memory.  The diagonals come bit-packed, a word per lane and layer (a set
// bit negates): as floats they were E scattered loads a lane (100k x 500: 11.5 ms).
template <typename CompT, bool QUERY, int E>
__global__ void __launch_bounds__(128)
encode_warp_kernel(const float* __restrict__ x, uint64_t n, int dim, int K, int rpb, const uint32_t* __restrict__ signbits /*[K][3][32]*/,
                   int flip_mask, CompT* __restrict__ codes, float* __restrict__ rotated, float* __restrict__ mags) {
    constexpr int P = 32 * E;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int first = E * lane;
    for (uint64_t row = uint64_t(blockIdx.x) * warps + warp; row < n; row += uint64_t(gridDim.x) * warps) {
        const float* src = x + row * uint64_t(dim);
        float in[E];
#pragma unroll
        for (int j = 0; j < E; ++j) in[j] = first + j < dim ? __ldg(src + first + j) : 0.0f;
        for (int r = blockIdx.y * rpb; r < min(K, int(blockIdx.y + 1) * rpb); ++r) {
            float v[E];
#pragma unroll
            for (int j = 0; j < E; ++j) v[j] = in[j];
            const uint32_t* sb = signbits + size_t(r) * 3 * 32 + lane;
#pragma unroll 1
            for (int layer = 0; layer < 3; ++layer) {
                const uint32_t word = __ldg(sb + layer * 32);
#pragma unroll
                for (int j = 0; j < E; ++j) v[j] = __uint_as_float(__float_as_uint(v[j]) ^ ((word << (31 - j)) & 0x80000000u));
#pragma unroll
                for (int h = 1; h < E; h <<= 1) {
#pragma unroll
                    for (int j = 0; j < E; ++j)
                        if ((j & h) == 0) {
                            const float a = v[j], b = v[j + h];
                            v[j] = __fadd_rn(a, b);
                            v[j + h] = __fsub_rn(a, b);
                        }
                }
#pragma unroll
                for (int t = 1; t < 32; t <<= 1) {
                    const bool upper = lane & t;
#pragma unroll
                    for (int j = 0; j < E; ++j) {
                        const float other = __shfl_xor_sync(0xffffffffu, v[j], t);
                        v[j] = upper ? __fsub_rn(other, v[j]) : __fadd_rn(v[j], other);
                    }
                }
            }
            // lowest-index argmax: ascending scan of the lane's own elements, then a warp reduction that prefers
            // the lower index on equal magnitude (cp_encoder.hpp:82-88)
            float best = -1.0f, win = 0.0f;
            int idx = 0x7fffffff;
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const float a = fabsf(v[j]);
                if (a > best) {
                    best = a;
                    win = v[j];
                    idx = first + j;
                }
            }
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) {
                const float ob = __shfl_xor_sync(0xffffffffu, best, o);
                const float ow = __shfl_xor_sync(0xffffffffu, win, o);
                const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
                if (ob > best || (ob == best && oi < idx)) {
                    best = ob;
                    win = ow;
                    idx = oi;
                }
            }
            if (lane == 0) {
                codes[row * K + r] = CompT(component_of(win, idx, flip_mask));
                if (QUERY && mags) mags[row * K + r] = best;
            }
            if (QUERY && rotated) {
                float* out = rotated + (row * K + r) * uint64_t(P) + first;
#pragma unroll
                for (int j = 0; j < E; ++j) out[j] = (__popc((first + j) & flip_mask) & 1) ? -v[j] : v[j];
            }
        }
    }
}

// ---- padded dims 256, 512, many vectors: G = 2, 4 lanes per vector, 128 elements per lane ---------------------------
// What bounds it is the add pipe, with the shuffles beside it.  With 128 elements a lane only g = log2(G) of the
// log2(P) stages of a layer reach across lanes.  They become register stages too: a swap of an element bit that the
// lanes carry with one that the registers carry moves half of the registers, one shuffle for each.
//   The register of index r (7 bits) holds the element whose low 7 - g bits are r's and whose next g bits, or top g
// bits, are r's top g bits XOR the lane's index in its group; the lane's index is the other of the two.  So every lane
// sends the registers whose bit i is set to the lane whose bit i differs, and stores what it gets where it came from:
// no selects.  In the butterflies over those bits a lane whose bit is set holds the operands the other way round,
//     v[p] = s v[p] + v[q],  v[q] = v[p] - s v[q],  s = +-1 by lane,
// which is x + y and x - y with one rounding each, as the reference has them.
//   A layer starts with the top bits in the lanes (the first) or the middle ones (the later ones, as the layer before
// left them).  Against a warp a vector with a shuffle for every element and stage across lanes: 100k x 500, K = 32, 4.26 ms
// -> 2.46; 100k x 256, 2.08 -> 1.13.  (At 1024, eight lanes a vector, 5.9 ms against the transposes' 5.3.)
template <int G>
__device__ __forceinline__ void swap_bits(f32x2 (&v)[64]) {
    constexpr int kSwap = G == 2 ? 1 : 2;
#pragma unroll
    for (int i = 0; i < kSwap; ++i) {
#pragma unroll
        for (int p = 0; p < 64; ++p)
            if (p & (64 >> kSwap) << i) {
                float a, b;
                unpack2(v[p], a, b);
                v[p] = pack2(__shfl_xor_sync(0xffffffffu, a, 1 << i), __shfl_xor_sync(0xffffffffu, b, 1 << i));
            }
    }
}

// the g stages over the registers' top bits
template <int G>
__device__ __forceinline__ void swapped_stages(f32x2 (&v)[64], int part) {
    constexpr int kSwap = G == 2 ? 1 : 2;
#pragma unroll
    for (int i = 0; i < kSwap; ++i) {
        const float s = (part >> i & 1) ? -1.0f : 1.0f;
        const f32x2 plus = pack2(s, s), minus = pack2(-s, -s);
        const int h = (64 >> kSwap) << i;
#pragma unroll
        for (int p = 0; p < 64; ++p)
            if (!(p & h)) {
                const f32x2 a = v[p], b = v[p + h];
                v[p] = fma2(a, plus, b);
                v[p + h] = fma2(b, minus, a);
            }
    }
}

template <typename CompT, bool QUERY, int G>
__global__ void __launch_bounds__(kTileVecs, QUERY ? 2 : 3)
encode_group_kernel(const float* __restrict__ x, uint64_t n, int dim, int K, int rpb, const uint4* __restrict__ signbits /*[K][3][G]*/,
                    int flip_mask, CompT* __restrict__ codes, float* __restrict__ rotated, float* __restrict__ mags) {
    constexpr int kSwap = G == 2 ? 1 : 2, kLow = 7 - kSwap, kVecs = kTileVecs / G, kStride = kTileStride<128>;
    extern __shared__ float smem[];
    float* tile = smem;                                                     // [kTileVecs][kStride], 128 elements a row
    CompT* code_tile = reinterpret_cast<CompT*>(tile + kTileVecs * kStride);  // [kVecs][rotations of this block]
    const int r0 = blockIdx.y * rpb, r1 = min(K, r0 + rpb), nr = r1 - r0;
    const uint64_t row0 = uint64_t(blockIdx.x) * kVecs;
    const int rows = int(min(uint64_t(kVecs), n - row0));
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, part = t % G;

    stage_tile<128 * G>(tile, x, row0, rows, dim, lane, warp);
    __syncthreads();

    const f32x2* mine = reinterpret_cast<const f32x2*>(tile + t * kStride);
    const uint64_t row = row0 + t / G;
    const uint4* sb = signbits + size_t(r0) * 3 * G + part;
    uint4 next = __ldg(sb);
    for (int r = r0; r < r1; ++r) {
        f32x2 v[64];
#pragma unroll
        for (int p = 0; p < 64; ++p) v[p] = mine[p ^ part << (kLow - 1)];
#pragma unroll 1
        for (int layer = 0; layer < 3; ++layer) {
            const uint4 sign = next;
            sb += G;
            if (r + 1 < r1 || layer < 2) next = __ldg(sb);
#pragma unroll
            for (int p = 0; p < 64; ++p) {
                const uint32_t word = p < 16 ? sign.x : (p < 32 ? sign.y : (p < 48 ? sign.z : sign.w));
                float a, b;
                unpack2(v[p], a, b);
                a = __uint_as_float(__float_as_uint(a) ^ ((word << (31 - 2 * (p & 15))) & 0x80000000u));
                b = __uint_as_float(__float_as_uint(b) ^ ((word << (30 - 2 * (p & 15))) & 0x80000000u));
                v[p] = pack2(__fadd_rn(a, b), __fsub_rn(a, b));
            }
            butterfly_stages<1, 64, 1 << (kLow - 1)>(v);
            if (layer > 0) swap_bits<G>(v);
            swapped_stages<G>(v, part);
            swap_bits<G>(v);
            swapped_stages<G>(v, part);
        }
        // the lowest index of the largest magnitude: a left-biased tournament in the order of the element bits, the
        // sides of the top ones changed in the lanes that hold them the other way round; then across the lanes
        float best, win;
        int idx;
        {
            float w[64];
            int id[64];
#pragma unroll
            for (int p = 0; p < 64; ++p) {
                float a, b;
                unpack2(v[p], a, b);
                const bool right = fabsf(b) > fabsf(a);
                w[p] = right ? b : a;
                id[p] = right ? 2 * p + 1 : 2 * p;
            }
#pragma unroll
            for (int m = 32; m >= 1; m >>= 1) {
                const bool turned = m <= (64 >> kLow) && (part & (64 >> kLow) / m);
#pragma unroll
                for (int p = 0; p < m; ++p) {
                    const float a = fabsf(w[2 * p]), b = fabsf(w[2 * p + 1]);
                    const bool right = b > a || (turned && b == a);
                    w[p] = right ? w[2 * p + 1] : w[2 * p];
                    id[p] = right ? id[2 * p + 1] : id[2 * p];
                }
            }
            win = w[0], best = fabsf(win);
            idx = (id[0] & ((1 << kLow) - 1)) | part << kLow | ((id[0] >> kLow) ^ part) << 7;
        }
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const float ow = __shfl_xor_sync(0xffffffffu, win, o);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
            if (fabsf(ow) > best || (fabsf(ow) == best && oi < idx)) {
                best = fabsf(ow);
                win = ow;
                idx = oi;
            }
        }
        if (part == 0) code_tile[t / G * nr + (r - r0)] = CompT(component_of(win, idx, flip_mask));
        if (QUERY) {
            if (mags && part == 0 && t / G < rows) mags[row * K + r] = best;
            if (rotated) {
                swap_bits<G>(v);  // back to 128 consecutive elements a lane
                if (t / G < rows) {
                    float4* out = reinterpret_cast<float4*>(rotated + (row * K + r) * uint64_t(128 * G)) + 32 * part;
#pragma unroll
                    for (int c = 0; c < 32; ++c) {
                        float a0, a1, a2, a3;
                        unpack2(v[2 * c], a0, a1);
                        unpack2(v[2 * c + 1], a2, a3);
                        float4 o;
                        o.x = (__popc((4 * c) & flip_mask) & 1) ? -a0 : a0;
                        o.y = (__popc((4 * c + 1) & flip_mask) & 1) ? -a1 : a1;
                        o.z = (__popc((4 * c + 2) & flip_mask) & 1) ? -a2 : a2;
                        o.w = (__popc((4 * c + 3) & flip_mask) & 1) ? -a3 : a3;
                        out[c ^ part << (kLow - 2)] = o;
                    }
                }
            }
        }
    }
    __syncthreads();
    CompT* dst = codes + row0 * uint64_t(K);
    if (nr == K) {
        for (int i = t; i < rows * K; i += kTileVecs) dst[i] = code_tile[i];
    } else {
        for (int i = t; i < rows * nr; i += kTileVecs) dst[uint64_t(i / nr) * K + r0 + i % nr] = code_tile[i];
    }
}

// ---- generic padded dim: one warp per vector, transform in shared memory ----------------------
template <typename CompT>
__global__ void encode_generic_kernel(const float* __restrict__ x, uint64_t n, int dim, int P, int K,
                                      const float* __restrict__ signs /*[K][3][P]*/, int flip_mask,
                                      CompT* __restrict__ codes, float* __restrict__ rotated,
                                      float* __restrict__ mags) {
    extern __shared__ float smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    float* buf = smem + size_t(warp) * P;
    for (uint64_t row = uint64_t(blockIdx.x) * warps + warp; row < n; row += uint64_t(gridDim.x) * warps) {
        const float* src = x + row * uint64_t(dim);
        for (int r = 0; r < K; ++r) {
            const float* sg = signs + size_t(r) * 3 * P;
            for (int layer = 0; layer < 3; ++layer) {
                // diagonal (layer 0 also loads and zero-pads)
                for (int i = lane; i < P; i += 32) {
                    float a = layer == 0 ? (i < dim ? __ldg(src + i) : 0.0f) : buf[i];
                    buf[i] = __fmul_rn(a, sg[layer * P + i]);
                }
                __syncwarp();
                for (int h = 1; h < P; h <<= 1) {
                    for (int b = lane; b < P / 2; b += 32) {
                        int j = ((b / h) * 2 * h) + (b % h);
                        float a = buf[j], c = buf[j + h];
                        buf[j] = __fadd_rn(a, c);
                        buf[j + h] = __fsub_rn(a, c);
                    }
                    __syncwarp();
                }
            }
            // lowest-index argmax: strided scan per lane (ascending index), then a warp
            // reduction that prefers the lower index on equal magnitude
            float best = -1.0f, win = 0.0f;  // -1: the first element a lane sees always wins
            int idx = 0x7fffffff;
            for (int i = lane; i < P; i += 32) {
                float a = fabsf(buf[i]);
                if (a > best) {
                    best = a;
                    win = buf[i];
                    idx = i;
                }
            }
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) {
                float ob = __shfl_xor_sync(0xffffffffu, best, o);
                float ow = __shfl_xor_sync(0xffffffffu, win, o);
                int oi = __shfl_xor_sync(0xffffffffu, idx, o);
                if (ob > best || (ob == best && oi < idx)) {
                    best = ob;
                    win = ow;
                    idx = oi;
                }
            }
            if (lane == 0) {
                codes[row * K + r] = CompT(component_of(win, idx, flip_mask));
                if (mags) mags[row * K + r] = best;
            }
            if (rotated) {
                float* out = rotated + (row * K + r) * uint64_t(P);
                for (int i = lane; i < P; i += 32)
                    out[i] = (__popc(i & flip_mask) & 1) ? -buf[i] : buf[i];
            }
            __syncwarp();
        }
    }
}

}  // namespace

// binary-code mode: every component reduced to its sign bit; 32-bit words where the buffer allows
__global__ void sign_only_kernel(uint32_t* __restrict__ codes, uint64_t words, uint32_t mask) {
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < words) codes[i] &= mask;
}
__global__ void sign_only_bytes_kernel(unsigned char* __restrict__ codes, uint64_t bytes, int comp_bytes) {
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < bytes) codes[i] &= (comp_bytes == 2 && (i & 1)) ? 0u : 1u;  // little-endian halfwords: the high byte is cleared
}

// The rotations of a vector are independent, so few vectors spread them over blocks until `want` blocks are in flight
// (a lone vector of padded dim 128: one thread's 32 rotations in sequence took 115 us, one rotation a block 7 us).
static int rotations_per_block(uint64_t blocks, uint64_t want, int K) {
    uint64_t split = (want + blocks - 1) / blocks;
    if (split > uint64_t(K)) split = K;
    return int((K + split - 1) / split);
}

uint32_t p1024_element(int layer, int lane, int reg) {
    return uint32_t(index_part(reg, 0, 3 * layer) | index_part(lane, 5, 3 * layer));
}

int launch_encode(cphnsw_b200_index* h, const float* d_x, uint64_t n, void* d_codes, float* d_rot,
                  float* d_mag, cudaStream_t st) {
    if (n == 0) return 0;
    const int P = int(h->P), K = int(h->K), dim = int(h->dim);
    // width of the reference's in-register SIMD phase for this build and length
    // (fht.hpp:141-147: AVX-512 defers to AVX2 below 16; :81-87: AVX2 defers to scalar below 8)
    int w = 1;
    if (h->convention == CPHNSW_B200_FHT_AVX512 && P >= 16) w = 16;
    else if (h->convention >= CPHNSW_B200_FHT_AVX2 && P >= 8) w = 8;
    const int flip_mask = w - 1;
    const float* signs = h->d_signs.as<float>();
    LaunchTimer timer(h, kKernelEncode, st);
    const bool query = d_rot || d_mag;
    // (a buffer for the rotated vectors off a 16-byte boundary: the kernels with scalar stores)
    const bool wide = (reinterpret_cast<uintptr_t>(d_rot) & 15) == 0;
    // 256 and 512: lanes in groups from two to four blocks an SM on; fewer vectors leave most of a group's long chain of
    // instructions exposed (one of 256: 10.7 us against 6.6; 1,000: 31 against 29; 500 of 512: 33 against 41).  Rotated
    // vectors of 256 stay with the warp kernel, whose stores are whole lines (2,000: 58 us against 65).
    const uint64_t group_tiles = (P == 512 && wide) || (P == 256 && !query) ? (n * (P / 128) + kTileVecs - 1) / kTileVecs : 0;

    if (P == 32 || P == 64 || (P == 128 && wide)) {
        const uint64_t tiles = (n + kTileVecs - 1) / kTileVecs;
        const int rpb = rotations_per_block(tiles, uint64_t(h->sm_count) * (P == 128 ? 6 : 12), K);
        const size_t smem = size_t(kTileVecs) * (P + 2) * sizeof(float) + size_t(2) * 3 * P * sizeof(float) + size_t(kTileVecs) * rpb * h->comp_bytes;
        const dim3 grid(unsigned(tiles), unsigned((K + rpb - 1) / rpb));
#define CPB_LAUNCH_THREAD(T, Q, PP)                                                                        \
    do {                                                                                                   \
        CPB_CUDA(allow_max_dynamic_smem(encode_thread_kernel<T, Q, PP>));                                  \
        encode_thread_kernel<T, Q, PP><<<grid, kTileVecs, smem, st>>>(d_x, n, dim, K, rpb, signs, flip_mask, \
                                                                     (T*)d_codes, d_rot, d_mag);            \
    } while (0)
#define CPB_LAUNCH_THREAD_P(T, Q)                       \
    do {                                                \
        if (P == 32) CPB_LAUNCH_THREAD(T, Q, 32);       \
        else if (P == 64) CPB_LAUNCH_THREAD(T, Q, 64);  \
        else CPB_LAUNCH_THREAD(T, Q, 128);              \
    } while (0)
        if (h->comp_bytes == 1) {
            if (query) CPB_LAUNCH_THREAD_P(uint8_t, true);
            else CPB_LAUNCH_THREAD_P(uint8_t, false);
        } else {
            if (query) CPB_LAUNCH_THREAD_P(uint16_t, true);
            else CPB_LAUNCH_THREAD_P(uint16_t, false);
        }
#undef CPB_LAUNCH_THREAD_P
#undef CPB_LAUNCH_THREAD
    } else if (P == kP1024 && h->d_signbits.p) {
        const uint64_t blocks = (n + kWarps1024 - 1) / kWarps1024;
        const int rpb = rotations_per_block(blocks, uint64_t(h->sm_count) * 16, K);
        // (many vectors: as many blocks as are resident)
        const uint64_t most = uint64_t(h->sm_count) * kBlocks1024;
        const dim3 grid(unsigned(blocks < most ? blocks : most), unsigned((K + rpb - 1) / rpb));
        const uint32_t* sb = h->d_signbits.as<uint32_t>();
#define CPB_LAUNCH_P1024(T, Q)                                                                              \
    encode_p1024_kernel<T, Q><<<grid, kWarps1024 * 32, 0, st>>>(d_x, n, dim, K, rpb, sb, flip_mask, (T*)d_codes, d_rot, d_mag)
        if (h->comp_bytes == 1) {  // (a 1-byte component cannot hold a 1024-wide index; kept for symmetry)
            if (query) CPB_LAUNCH_P1024(uint8_t, true);
            else CPB_LAUNCH_P1024(uint8_t, false);
        } else {
            if (query) CPB_LAUNCH_P1024(uint16_t, true);
            else CPB_LAUNCH_P1024(uint16_t, false);
        }
#undef CPB_LAUNCH_P1024
    } else if (group_tiles * K >= uint64_t(h->sm_count) * (P == 256 ? 4 : 2)) {
        const int vecs = kTileVecs / (P / 128);
        const uint64_t tiles = group_tiles;
        const int rpb = rotations_per_block(tiles, uint64_t(h->sm_count) * 6, K);
        const size_t smem = size_t(kTileVecs) * kTileStride<128> * sizeof(float) + size_t(vecs) * rpb * h->comp_bytes;
        const dim3 grid(unsigned(tiles), unsigned((K + rpb - 1) / rpb));
        const uint4* sb = h->d_signbits.as<uint4>() + kWarpSignWords / 4 * K;
#define CPB_LAUNCH_GROUP(T, Q, G)                                                                       \
    do {                                                                                                \
        CPB_CUDA(allow_max_dynamic_smem(encode_group_kernel<T, Q, G>));                                 \
        encode_group_kernel<T, Q, G><<<grid, kTileVecs, smem, st>>>(d_x, n, dim, K, rpb, sb, flip_mask, \
                                                                    (T*)d_codes, d_rot, d_mag);         \
    } while (0)
#define CPB_LAUNCH_GROUP_P(T)                       \
    do {                                            \
        if (P == 256) CPB_LAUNCH_GROUP(T, false, 2);  \
        else if (query) CPB_LAUNCH_GROUP(T, true, 4); \
        else CPB_LAUNCH_GROUP(T, false, 4);         \
    } while (0)
        if (h->comp_bytes == 1) CPB_LAUNCH_GROUP_P(uint8_t);  // binary codes keep the sign bits only
        else CPB_LAUNCH_GROUP_P(uint16_t);
#undef CPB_LAUNCH_GROUP_P
#undef CPB_LAUNCH_GROUP
    } else if (P == 256 || P == 512) {
        const uint32_t* sb = h->d_signbits.as<uint32_t>();
        const uint64_t blocks = (n + 3) / 4;
        const int rpb = rotations_per_block(blocks, uint64_t(h->sm_count) * 32, K);
        const dim3 grid(unsigned(blocks < uint64_t(h->sm_count) * 32 ? blocks : uint64_t(h->sm_count) * 32), unsigned((K + rpb - 1) / rpb));
#define CPB_LAUNCH_WARP(T, Q, EE) \
    encode_warp_kernel<T, Q, EE><<<grid, 128, 0, st>>>(d_x, n, dim, K, rpb, sb, flip_mask, (T*)d_codes, d_rot, d_mag)
#define CPB_LAUNCH_WARP_E(T, Q)                      \
    do {                                             \
        if (P == 256) CPB_LAUNCH_WARP(T, Q, 8);      \
        else CPB_LAUNCH_WARP(T, Q, 16);              \
    } while (0)
        if (h->comp_bytes == 1) {
            if (query) CPB_LAUNCH_WARP_E(uint8_t, true);
            else CPB_LAUNCH_WARP_E(uint8_t, false);
        } else {
            if (query) CPB_LAUNCH_WARP_E(uint16_t, true);
            else CPB_LAUNCH_WARP_E(uint16_t, false);
        }
#undef CPB_LAUNCH_WARP_E
#undef CPB_LAUNCH_WARP
    } else {
        int warps = 4;
        while (warps > 1 && size_t(warps) * P * sizeof(float) > 96 * 1024) warps >>= 1;
        size_t smem = size_t(warps) * P * sizeof(float);
        uint64_t blocks = (n + warps - 1) / warps;
        unsigned grid = unsigned(blocks < uint64_t(h->sm_count) * 16 ? blocks : uint64_t(h->sm_count) * 16);
        if (h->comp_bytes == 1) {
            CPB_CUDA(allow_max_dynamic_smem(encode_generic_kernel<uint8_t>));
            encode_generic_kernel<uint8_t><<<grid, warps * 32, smem, st>>>(d_x, n, dim, P, K, signs, flip_mask,
                                                                          (uint8_t*)d_codes, d_rot, d_mag);
        } else {
            CPB_CUDA(allow_max_dynamic_smem(encode_generic_kernel<uint16_t>));
            encode_generic_kernel<uint16_t><<<grid, warps * 32, smem, st>>>(d_x, n, dim, P, K, signs, flip_mask,
                                                                           (uint16_t*)d_codes, d_rot, d_mag);
        }
    }
    h->launches++;
    CPB_CUDA(cudaGetLastError());
    if (h->binary_codes && d_codes) {
        // binary-code mode: a component keeps only its sign bit (the unified encoder's primary code,
        // include/cphnsw/encoder/cp_encoder.hpp:165-176)
        const uint64_t bytes = n * uint64_t(K) * h->comp_bytes;
        if ((reinterpret_cast<uintptr_t>(d_codes) & 3) == 0 && (bytes & 3) == 0)
            sign_only_kernel<<<unsigned((bytes / 4 + 255) / 256), 256, 0, st>>>(static_cast<uint32_t*>(d_codes), bytes / 4,
                                                                              h->comp_bytes == 2 ? 0x00010001u : 0x01010101u);
        else
            sign_only_bytes_kernel<<<unsigned((bytes + 255) / 256), 256, 0, st>>>(static_cast<unsigned char*>(d_codes), bytes,
                                                                                 int(h->comp_bytes));
        h->launches++;
        CPB_CUDA(cudaGetLastError());
    }
    return 0;
}

}  // namespace cpb
