// Brute-force code-distance kNN graph with the tensor cores as a filter.
//
// Same result as the two other kNN kernels (k smallest under (distance, id), self excluded).  The distance of two codes
// is K minus the number of components they share.  Every component is hashed to one of S = 8 (K <= 32) or 4 symbols and a
// symbol is written as a row of the S-point Hadamard matrix without its constant column: S - 1 values of +-1 whose dot
// product is S - 1 for equal symbols and -1 for different ones.  The dot product of two such rows of (S - 1) K values is
// S m - K, m the number of components with equal symbols, and m is at least the number of equal components: a pair whose
// dot product is below S (K - t) - K differs in more than t components.  The products run on tcgen05 in fp8 with fp16
// accumulators (+-1 and integers up to 224 are exact in both), so all n^2 pairs cost 2 * 224 tensor operations and one
// instruction of the epilogue each; only pairs that reach the row's threshold t have their exact distance computed.
//
// Row thresholds.  Before the sweep a bound is taken from likely neighbours: rows sorted by two of their components lie
// beside rows that share both, and the k-th smallest exact distance in the windows of 128 around a row in eight such
// orders, every row counted once, bounds its final t from above.  On clustered data t is mostly right or one too high, and
// some 450 pairs per row pass, 140 of them truly within t.  The pairs found are kept in a buffer; when it runs full its k
// best are kept and t falls below the worst of them for the pairs still to come, which have higher ids.  On data without
// clusters the bound says nothing, t is lowered by this alone and most pairs pass: a sample of the data shows it, and the
// sweep is then left to another kernel ("what the filter is worth" below).
//
// Shape.  A block owns 256 rows, their operand resident in shared memory (56 KB at 224 values), and sweeps the candidates
// in tiles of 256, two stages of bulk copies.  A tile is two groups of tcgen05.mma with M = 128, N = 256 into the two
// halves of tensor memory; while one half is computed the other is read.  A row has two epilogue threads, which take the
// tiles in turn (a buffer and a limit each): one reads a tile while the other still deals with the pairs of the one before.
// The operand is laid out by the expansion kernel in the form the tensor core reads (8-row by 16-byte core matrices), so a
// tile is one contiguous copy and no tensor map is needed.  Blocks that take whole rows of tiles sweep them in step, so
// that a tile comes from L2; only the rows left over by the last full wave are split between blocks along the candidates.
#include <cuda_fp16.h>

#include "mma_common.cuh"

namespace cpb {
namespace {

using knn::kFull;
using knn::kWaitLimit;
using knn::mbar_wait_bounded;
using knn::smem_u32;
using namespace mma;

constexpr int kMmaCap = 384;              // entries of a buffer: at most 128 before a tile and 256 from it
constexpr int kMmaSlots = kMmaCap / 32;   // of them per lane
constexpr uint32_t kMmaKeep = 128;
constexpr int kEpiWarps = 16;             // epilogue warps: a quarter of the lanes, a half of the rows, every second tile
constexpr int kMmaThreads = (kEpiWarps + 3) * 32;  // and one each for the operands' copies, the products, the codes' copies
constexpr int kMaxCodeStages = 4;
constexpr size_t kMmaSmem = 216 * 1024;   // dynamic shared memory a block may use beside its 9 KB of static
constexpr int kBoundOrders = 8;           // orders of likely neighbours
constexpr int kBoundWindow = 128;         // rows looked at per order
constexpr uint32_t kKeys = 65536;

// symbols and values of a code shape; 0 symbols: not served
struct HashShape {
    int symbols, chunks;  // chunks: 16-byte pieces of a row's operand, an even number
};
__host__ __device__ inline HashShape hash_shape(int K) {
    HashShape s;
    s.symbols = K <= 32 ? 8 : (K <= 64 ? 4 : 0);
    const int values = K * (s.symbols - 1);
    s.chunks = (values + 31) / 32 * 2;
    return s;
}

__device__ __forceinline__ uint32_t symbol_of(uint32_t comp, uint32_t symbols) {
    return (comp ^ (comp >> 3) ^ (comp >> 6) ^ (comp >> 9)) & (symbols - 1);
}

// ---- operand: [tile of 256 rows][chunk][row][16 values] ------------------------------------------------------------
template <typename CompT>
__global__ void expand_codes_kernel(const CompT* __restrict__ codes, uint64_t n, int K, int symbols, int chunks,
                                    uint4* __restrict__ out, uint64_t tiles, SweepChoice choice) {
    if (choice.skip()) return;
    const uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= tiles * chunks * kMmaRows) return;
    const int r = int(t % kMmaRows), c = int(t / kMmaRows % chunks);
    const uint64_t row = t / (uint64_t(kMmaRows) * chunks) * kMmaRows + r;
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (row < n) {
        int comp = c * 16 / (symbols - 1), j = c * 16 % (symbols - 1) + 1;
        uint32_t h = comp < K ? symbol_of(codes[row * K + comp], uint32_t(symbols)) : 0u;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const uint32_t e4m3 = (__popc(h & uint32_t(j)) & 1) ? 0xB8u : 0x38u;  // -1 : +1
            if (comp < K) w[i / 4] |= e4m3 << (8 * (i % 4));
            if (++j == symbols) {
                j = 1;
                ++comp;
                if (comp < K) h = symbol_of(codes[row * K + comp], uint32_t(symbols));
            }
        }
    }
    out[t] = make_uint4(w[0], w[1], w[2], w[3]);
}

// ---- exact distance: differing bytes / halfwords of two padded rows -------------------------------------------------
// a flag in the top bit of every differing byte (halfword), the flags of 8 (16) words packed for one popcount
template <bool U16, int QUADS>
__device__ __forceinline__ uint32_t code_distance(const uint4* a, const uint4* b) {
    constexpr uint32_t LO = U16 ? 0x7fff7fffu : 0x7f7f7f7fu;
    constexpr int G = U16 ? 16 : 8;
    uint32_t d = 0, acc = 0;
#pragma unroll
    for (int i = 0; i < QUADS; ++i) {
        const uint4 x = a[i], y = b[i];
        const uint32_t v[4] = {x.x ^ y.x, x.y ^ y.y, x.z ^ y.z, x.w ^ y.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int sh = (i * 4 + j) % G;
            acc |= ((((v[j] & LO) + LO) | v[j]) >> sh) & (~LO >> sh);
        }
        if ((i + 1) * 4 % G == 0 || i + 1 == QUADS) {
            d += __popc(acc);
            acc = 0;
        }
    }
    return d;
}

// Smallest T with at least `need` of the lanes' entries at distance <= T (entries without a node hold kFull); K when
// there are fewer.
template <int SLOTS>
__device__ __forceinline__ uint32_t kth_distance(const uint32_t (&dist)[SLOTS], uint32_t need, int K) {
    uint32_t lo = 0, hi = uint32_t(K);
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        uint32_t c = 0;
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) c += dist[s] <= mid;
        if (__reduce_add_sync(kFull, c) >= need) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// the same over distances packed as bytes, entries without a node 127 (distances are 64 at most)
template <int WORDS>
__device__ __forceinline__ uint32_t count_upto(const uint32_t (&dist)[WORDS], uint32_t d) {
    const uint32_t top = d * 0x01010101u | 0x80808080u;  // less a byte of d or below: the flag stays
    uint32_t c = 0;
#pragma unroll
    for (int w = 0; w < WORDS; ++w) c += __popc((top - dist[w]) & 0x80808080u);
    return __reduce_add_sync(kFull, c);
}
template <int WORDS>
__device__ __forceinline__ uint32_t kth_packed(const uint32_t (&dist)[WORDS], uint32_t need, int K) {
    uint32_t lo = 0, hi = uint32_t(K);
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (count_upto(dist, mid) >= need) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// ---- bounds from likely neighbours ---------------------------------------------------------------------------------
// the low 8 bits of two components (the sign and the low index bits; all of a one-byte component)
template <typename CompT>
__device__ __forceinline__ uint32_t row_key(const CompT* codes, int K, uint64_t row, int order) {
    return (uint32_t(codes[row * K + (2 * order) % K]) & 0xffu) << 8 | (uint32_t(codes[row * K + (2 * order + 1) % K]) & 0xffu);
}
template <typename CompT>
__global__ void key_count_kernel(const CompT* __restrict__ codes, uint64_t n, int K, uint32_t* __restrict__ hist) {
    const uint64_t row = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (row < n) atomicAdd(hist + size_t(blockIdx.y) * kKeys + row_key(codes, K, row, blockIdx.y), 1u);
}
// exclusive, one block per order; a warp takes 2,048 keys, 128 of them a step in one line of reads each (a thread with 64
// keys of its own read a sector per key pair: 30 us)
__global__ void __launch_bounds__(1024) key_scan_kernel(uint32_t* __restrict__ hist) {
    __shared__ uint32_t sums[32];
    constexpr int kSteps = int(kKeys / 4096);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint4* h = reinterpret_cast<uint4*>(hist + size_t(blockIdx.x) * kKeys) + warp * kSteps * 32 + lane;
    auto scan = [&](uint32_t x) {  // inclusive, over the lanes
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, x, d);
            if (lane >= d) x += y;
        }
        return x;
    };
    uint32_t own = 0;
#pragma unroll
    for (int i = 0; i < kSteps; ++i) {
        const uint4 v = h[i * 32];
        own += v.x + v.y + v.z + v.w;
    }
    own = __reduce_add_sync(kFull, own);
    if (lane == 0) sums[warp] = own;
    __syncthreads();
    if (warp == 0) {
        const uint32_t o = sums[lane];
        sums[lane] = scan(o) - o;
    }
    __syncthreads();
    uint32_t at = sums[warp];
#pragma unroll 4
    for (int i = 0; i < kSteps; ++i) {
        const uint4 c = h[i * 32];
        const uint32_t mine = c.x + c.y + c.z + c.w, upto = scan(mine), b = at + upto - mine;
        h[i * 32] = make_uint4(b, b + c.x, b + c.x + c.y, b + c.x + c.y + c.z);
        at += __shfl_sync(kFull, upto, 31);
    }
}
template <typename CompT>
__global__ void key_scatter_kernel(const CompT* __restrict__ codes, uint64_t n, int K, uint32_t* __restrict__ hist,
                                   uint32_t* __restrict__ order /* [orders][n] */, uint32_t* __restrict__ place /* [n][orders] */) {
    const uint64_t row = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (row >= n) return;
    const uint32_t at = atomicAdd(hist + size_t(blockIdx.y) * kKeys + row_key(codes, K, row, blockIdx.y), 1u);
    order[size_t(blockIdx.y) * n + at] = uint32_t(row);
    place[row * kBoundOrders + blockIdx.y] = at;
}
// a row of QUADS 16-byte words; SECTORS: two words by one instruction, the row 32-byte aligned
template <bool SECTORS, int QUADS>
__device__ __forceinline__ void load_row(uint4 (&v)[QUADS], const uint4* p) {
    if constexpr (SECTORS) {
#pragma unroll
        for (int w = 0; w < QUADS; w += 2)
            asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=r"(v[w].x), "=r"(v[w].y), "=r"(v[w].z), "=r"(v[w].w), "=r"(v[w + 1].x), "=r"(v[w + 1].y), "=r"(v[w + 1].z),
                           "=r"(v[w + 1].w)
                         : "l"(p + w));
    } else {
#pragma unroll
        for (int w = 0; w < QUADS; ++w) v[w] = __ldg(p + w);
    }
}
// A warp takes a row: the k-th smallest distance among the rows in the windows around it in all orders, each counted
// once.  (The least of the orders' own k-th distances is 0.4 to 1 higher, which lets half as many pairs again through.)
// Rows are taken as the first order has them, whose neighbours share much of their windows.
// What bounds it is the gather of 1,024 code rows through the L1, and registers in flight: distances are packed as bytes
// (half the work of counting them, 24 registers less) and a 32-byte row is one load where it is aligned.  100k rows, K = 32:
// 1.15 ms before, 0.85 now with one-byte components, 1.66 and 1.32 with two-byte ones.
constexpr int kBoundWarps = 4;
constexpr uint32_t kSeenSlots = 1024;
template <bool U16, int QUADS, bool SECTORS>
__global__ void __launch_bounds__(kBoundWarps * 32)
bound_kernel(const uint4* __restrict__ codes, int K, uint64_t n, const uint32_t* __restrict__ order, const uint32_t* __restrict__ place,
             uint32_t k, uint32_t row_begin, uint32_t row_end, uint32_t* __restrict__ bound, uint64_t apart /* of LoadArgs: its rows only; 0: all rows */,
             SweepChoice choice) {
    if (choice.skip()) return;
    constexpr int S = kBoundWindow / 32, N = kBoundOrders * S;
    __shared__ uint32_t seen_sm[kBoundWarps][kSeenSlots];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t at = uint64_t(blockIdx.x) * kBoundWarps + warp;
    if (at >= n) return;
    const uint64_t wanted = apart ? row_begin + at / 32 * apart + at % 32 : order[at];
    if (wanted < row_begin || wanted >= row_end) return;
    const uint32_t row = uint32_t(wanted);
    uint32_t* seen = seen_sm[warp];
    for (uint32_t i = lane; i < kSeenSlots / 4; i += 32) reinterpret_cast<uint4*>(seen)[i] = make_uint4(kFull, kFull, kFull, kFull);
    const uint32_t where = lane < kBoundOrders ? place[uint64_t(row) * kBoundOrders + lane] : 0u;
    uint32_t id[N], dist[N / 4] = {};  // distances a byte each
    uint4 own[QUADS];
#pragma unroll
    for (int w = 0; w < QUADS; ++w) own[w] = __ldg(codes + size_t(row) * QUADS + w);
#pragma unroll
    for (int o = 0; o < kBoundOrders; ++o) {
        const uint64_t pos = __shfl_sync(kFull, where, o);
        uint64_t first = pos < kBoundWindow / 2 ? 0 : pos - kBoundWindow / 2;
        if (first + kBoundWindow > n) first = n > kBoundWindow ? n - kBoundWindow : 0;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const uint64_t p = first + s * 32 + lane;
            id[o * S + s] = p < n ? __ldg(order + size_t(o) * n + p) : row;
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        uint4 theirs[QUADS];
        load_row<SECTORS>(theirs, codes + size_t(id[i]) * QUADS);
        dist[i / 4] |= (id[i] != row ? code_distance<U16, QUADS>(own, theirs) : 127u) << (8 * (i % 4));
    }
    // enough of the closest, repeats included, to hold k different rows in most cases; half the table at most
    const uint32_t reach = kth_packed(dist, kSeenSlots / 2 < 4 * k ? kSeenSlots / 2 : 4 * k, K);
    const bool all = count_upto(dist, reach) <= kSeenSlots * 3 / 4;  // else the farthest of them would crowd the table
    __syncwarp();
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if ((dist[i / 4] >> (8 * (i % 4)) & 127u) < reach + (all ? 1u : 0u)) {
            uint32_t slot = (id[i] * 0x9E3779B1u) >> 22;
            while (true) {
                const uint32_t was = atomicCAS(seen + slot, kFull, id[i]);
                if (was == kFull) break;
                if (was == id[i]) {
                    dist[i / 4] |= 127u << (8 * (i % 4));  // a repeat
                    break;
                }
                slot = (slot + 1) & (kSeenSlots - 1);
            }
        } else {
            dist[i / 4] |= 127u << (8 * (i % 4));
        }
    }
    const uint32_t T = kth_packed(dist, k, K);  // (K when fewer than k were found)
    if (lane == 0) bound[row] = T;
}

// ---- what the filter is worth ----------------------------------------------------------------------------------------
// On clustered data next to nothing passes it, on data without clusters most pairs do (78 % at the final thresholds on
// 100k points of the unit sphere, K = 32), and the epilogue's warps spend a turn on every pair of the row that has most of
// them and one on every 32 of the 32 rows together.  Those turns are counted on a sample before anything else is done:
// kLoadGroups groups of 32 rows against kLoadTiles candidate tiles each, at the rows' bounds.  Above the caller's limit
// the sweep is left to another kernel.  (The share of pairs that would pass by chance at the bounds, which needs no pairs,
// tells less: mixtures of 1,000, 5,000 and 100 points a cluster with shares of 0.4, 0.0 and 3 % took 13, 9 and 26 ms.)
struct LoadArgs {
    uint64_t apart;  // groups of rows are so many rows apart
    uint32_t groups;
};
constexpr uint32_t kLoadGroups = 16, kLoadTiles = 16;

// the symbols of a word's components, in their places
template <bool U16>
__device__ __forceinline__ uint32_t symbols_of(uint32_t w, uint32_t symbols) {
    if (U16) return (w ^ (w >> 3 & 0x1fff1fffu) ^ (w >> 6 & 0x03ff03ffu) ^ (w >> 9 & 0x007f007fu)) & ((symbols - 1) * 0x00010001u);
    return (w ^ (w >> 3 & 0x1f1f1f1fu) ^ (w >> 6 & 0x03030303u)) & ((symbols - 1) * 0x01010101u);
}
// a block: 32 rows (their symbols in shared memory) against a tile, a candidate per thread
template <bool U16, int QUADS>
__global__ void __launch_bounds__(kMmaRows) load_kernel(const uint4* __restrict__ codes, uint64_t n, uint32_t symbols, uint32_t tiles,
                                                        uint32_t row_begin, uint32_t row_end, const uint32_t* __restrict__ bound, LoadArgs a,
                                                        unsigned long long* load) {
    __shared__ uint4 rows_sm[32][QUADS];
    __shared__ uint32_t bound_sm[32], passed[32];
    const uint32_t g = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const uint64_t row0 = row_begin + g * a.apart;
    const uint32_t have = uint32_t(row_end - row0 < 32 ? row_end - row0 : 32);
    const uint32_t tile = uint32_t((uint64_t(blockIdx.y) * a.groups + g) * tiles / (uint64_t(a.groups) * kLoadTiles));
    auto hashed = [&](uint4 v) {
        return make_uint4(symbols_of<U16>(v.x, symbols), symbols_of<U16>(v.y, symbols), symbols_of<U16>(v.z, symbols), symbols_of<U16>(v.w, symbols));
    };
    for (uint32_t i = tid; i < have * QUADS; i += kMmaRows) rows_sm[i / QUADS][i % QUADS] = hashed(__ldg(codes + row0 * QUADS + i));
    if (tid < 32) passed[tid] = 0, bound_sm[tid] = tid < have ? bound[row0 + tid] : 0u;
    const uint64_t col = uint64_t(tile) * kMmaRows + tid;
    uint4 own[QUADS];
#pragma unroll
    for (int w = 0; w < QUADS; ++w) own[w] = hashed(__ldg(codes + (col < n ? col : 0) * QUADS + w));
    __syncthreads();
    for (uint32_t r = 0; r < have; ++r) {
        const uint32_t m = __ballot_sync(kFull, col < n && code_distance<U16, QUADS>(rows_sm[r], own) <= bound_sm[r]);
        if (lane == 0 && m) atomicAdd(&passed[r], __popc(m));
    }
    __syncthreads();
    if (tid < 32) {
        const uint32_t most = __reduce_max_sync(kFull, passed[tid]), all = __reduce_add_sync(kFull, passed[tid]);
        if (tid == 0) atomicAdd(load, (unsigned long long)(most + (all + 31) / 32));
    }
}

// ---- tcgen05 pieces ------------------------------------------------------------------------------------------------
// D fp16, A and B e4m3, both K-major, M = 128, N = 256
constexpr uint32_t kIdesc = (uint32_t(256 >> 3) << 17) | (uint32_t(128 >> 4) << 24);

__device__ __forceinline__ void mma_f8(uint32_t d_tmem, uint64_t a, uint64_t b, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(kIdesc), "r"(uint32_t(accumulate))
        : "memory");
}
// 16 fp16 columns of the warp's 32 lanes of tensor memory, two neighbours per register: asked for, and waited for
__device__ __forceinline__ void tmem_load16(uint32_t (&r)[8], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.pack::16b.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr)
                 : "memory");
}
// (the registers are operands so that no use of them moves in front of the wait)
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])
                 :
                 : "memory");
}
struct KnnMmaArgs {
    const uint4* operand;  // [tiles][chunks][256]
    const uint4* codes;    // padded rows
    int code_stages;       // candidate tiles whose codes are held in shared memory
    int K, symbols, chunks;
    uint64_t n;
    uint32_t k;
    Split split;
    uint32_t tile0;               // first row tile of the launch
    uint32_t row_begin, row_end;  // rows wanted
    const uint32_t* bound;        // [n] bounds on the final thresholds
    uint32_t* ids;                // [segments][256 rows][2 sides][kMmaCap]
    uint8_t* dists;               // the same
    uint32_t* counts;             // [segments][256][2]
    uint32_t* status;
    uint32_t first_wait_polls, handover_polls;
    SweepChoice choice;
};

// A row tile's codes and limits pass between the two warps that share its rows: each stores, in shared memory, the number
// of segments it is done with, and waits for the other's before it replaces them.  (A counter and not a barrier's phase:
// a warp without a tile in a segment runs ahead of the other by several.)
__device__ __forceinline__ void hand_over(uint32_t* done, uint32_t segments) {
    asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_u32(done)), "r"(segments) : "memory");
}
__device__ __forceinline__ bool handed_over(const uint32_t* done, uint32_t segments, uint32_t limit, volatile int* aborted) {
    if (segments == 0) return true;
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t have;
        asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(have) : "r"(smem_u32(done)) : "memory");
        if (have >= segments) return true;
        if ((i & 15) == 15) {
            if (*aborted) return false;
            __nanosleep(200);
        }
    }
    return false;
}

// the dot product a pair at distance <= t reaches at least (t < 0: none does), twice
__device__ __forceinline__ __half2 dot_of_distance(int symbols, int K, int t) {
    return t < 0 ? __half2half2(__ushort_as_half(0x7c00)) : __float2half2_rn(float(symbols * (K - t) - K));
}

// The row's buffer shrinks to its k best (or all that are no worse than the k-th, up to kMmaKeep).  By the whole warp;
// returns the k-th distance and the new count.
__device__ __forceinline__ uint32_t compact_row(uint32_t* ids, uint8_t* dists, uint32_t& count, uint32_t k, int K, int lane) {
    uint32_t dist[kMmaSlots];
#pragma unroll
    for (int s = 0; s < kMmaSlots; ++s) {
        const uint32_t e = uint32_t(s * 32 + lane);
        dist[s] = e < count ? dists[e] : kFull;
    }
    const uint32_t T = kth_distance(dist, k, K);
    uint32_t below = 0, upto = 0;
#pragma unroll
    for (int s = 0; s < kMmaSlots; ++s) below += dist[s] < T, upto += dist[s] <= T;
    below = __reduce_add_sync(kFull, below);
    upto = __reduce_add_sync(kFull, upto);
    uint32_t last = kInvalidNode;  // largest id kept at distance T
    if (upto > kMmaKeep) {
        uint32_t lo = 0, hi = kInvalidNode;
        while (lo < hi) {
            const uint32_t mid = lo + ((hi - lo) >> 1);
            uint32_t c = 0;
#pragma unroll 1
            for (uint32_t e = lane; e < count; e += 32) c += dists[e] == T && ids[e] <= mid;
            if (__reduce_add_sync(kFull, c) >= k - below) hi = mid;
            else lo = mid + 1;
        }
        last = lo;
    }
    __syncwarp();
    uint32_t at = 0;
#pragma unroll 1
    for (uint32_t e = lane; e < (count + 31u) / 32 * 32; e += 32) {  // (an entry moves down or stays)
        const uint32_t d = e < count ? dists[e] : kFull, id = e < count ? ids[e] : kInvalidNode;
        const bool keep = d < T || (d == T && id <= last);
        const uint32_t m = __ballot_sync(kFull, keep);
        if (keep) {
            const uint32_t to = at + __popc(m & ((1u << lane) - 1u));
            ids[to] = id;
            dists[to] = uint8_t(d);
        }
        at += __popc(m);
        __syncwarp();
    }
    count = at;
    return T;
}

template <bool U16, int QUADS>  // QUADS: 16-byte words of a padded code row
__global__ void __launch_bounds__(kMmaThreads, 1) knn_mma_kernel(KnnMmaArgs a) {
    if (a.choice.skip()) return;
    extern __shared__ __align__(1024) unsigned char mma_smem[];
    __shared__ __align__(8) uint64_t full_bar[2][2], empty_bar[2][2];    // [stage][part of K]
    __shared__ __align__(8) uint64_t tfull_bar[2][2], tempty_bar[2][2];  // [half of the rows][side]
    __shared__ __align__(8) uint64_t cfull_bar[kMaxCodeStages], cempty_bar[kMaxCodeStages], drain_bar;
    __shared__ uint16_t queue[kEpiWarps][64];       // pairs a warp has collected: column | lane of the row << 8
    __shared__ uint32_t filled[2][kMmaRows];        // [side][row]: entries of the buffer
    __shared__ int limit[2][kMmaRows];              // [side][row]: largest distance still of use
    __shared__ uint32_t finished[kEpiWarps];        // segments the epilogue warps are done with
    __shared__ uint32_t tmem_base_sm;
    __shared__ int abort_flag;
    const int lane = threadIdx.x & 31, warp = __shfl_sync(kFull, int(threadIdx.x >> 5), 0);
    const uint32_t operand_bytes = uint32_t(a.chunks) * kMmaRows * 16;
    const int ksteps = a.chunks / 2, split_k = (ksteps + 1) / 2;  // 32 values of K a step: two 16-byte chunks
    unsigned char* a_sm = mma_smem;
    unsigned char* b_sm = mma_smem + operand_bytes;      // two stages
    unsigned char* c_sm = mma_smem + 3 * operand_bytes;  // the candidates' codes, code_stages of them
    constexpr uint32_t kCodeBytes = kMmaRows * QUADS * 16;
    constexpr uint32_t kStepBytes = 2 * kMmaRows * 16;
    constexpr bool kOwnInSmem = QUADS <= 4;  // the rows' own codes (wider ones: read from L2)
    const uint64_t s0 = a.split.first_step(blockIdx.x);
    const uint32_t steps = uint32_t(a.split.first_step(blockIdx.x + 1) - s0);
    const uint32_t rt0 = uint32_t(s0 / a.split.cts), ct0 = uint32_t(s0 % a.split.cts);  // first row and candidate tile

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i)
            for (int j = 0; j < 2; ++j) {
                knn::mbar_init(&full_bar[i][j], 1);
                knn::mbar_init(&empty_bar[i][j], 1);
                knn::mbar_init(&tfull_bar[i][j], 1);
                knn::mbar_init(&tempty_bar[i][j], 4);
            }
        for (int i = 0; i < kMaxCodeStages; ++i) {
            knn::mbar_init(&cfull_bar[i], 1);
            knn::mbar_init(&cempty_bar[i], kEpiWarps / 2);
        }
        knn::mbar_init(&drain_bar, 1);
        for (int i = 0; i < kEpiWarps; ++i) finished[i] = 0;
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kEpiWarps + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sm)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_sm;
    volatile int* aborted = &abort_flag;

    uint32_t loads = 0;  // copies issued by this warp: parts of operands, or code tiles
    if (warp == kEpiWarps) {
        if (lane == 0) {
            uint32_t rt = rt0, ct = ct0;
            bool fresh = true, ok = true;  // fresh: the row tile's own operand has to come too
            const unsigned char* op = reinterpret_cast<const unsigned char*>(a.operand);
            for (uint32_t i = 0; i < steps && ok && !*aborted; ++i) {
                const uint32_t s = i & 1;
                // a new row operand replaces the one that the step before still reads
                if (fresh && i) ok = wait_or_abort(&empty_bar[s ^ 1][1], ((i - 1) >> 1) & 1, kWaitLimit, aborted);
                for (int part = 0; part < 2 && ok; ++part) {
                    const uint32_t from = part ? split_k * kStepBytes : 0u;
                    const uint32_t bytes = (part ? ksteps - split_k : split_k) * kStepBytes;
                    ok = wait_or_abort(&empty_bar[s][part], ((i >> 1) & 1) ^ 1, kWaitLimit, aborted);
                    if (!ok) break;
                    const uint32_t own = fresh && part == 0 ? operand_bytes : 0u;
                    knn::mbar_expect_tx(&full_bar[s][part], bytes + own);
                    if (own) knn::bulk_g2s(a_sm, op + size_t(a.tile0 + rt) * operand_bytes, own, &full_bar[s][part]);
                    if (bytes) knn::bulk_g2s(b_sm + s * operand_bytes + from, op + size_t(ct) * operand_bytes + from, bytes, &full_bar[s][part]);
                    ++loads;
                }
                fresh = ++ct == a.split.cts;
                if (fresh) ct = 0, ++rt;
            }
            if (!ok) *aborted = 1;
        }
    } else if (warp == kEpiWarps + 2) {
        if (lane == 0) {
            uint32_t ct = ct0, cs = 0, parity = 1;
            for (uint32_t i = 0; i < steps && !*aborted; ++i) {
                if (!wait_or_abort(&cempty_bar[cs], parity, kWaitLimit, aborted)) {
                    *aborted = 1;
                    break;
                }
                const uint64_t left = a.n - uint64_t(ct) * kMmaRows;
                const uint32_t bytes = uint32_t(left < kMmaRows ? left : kMmaRows) * QUADS * 16;
                knn::mbar_expect_tx(&cfull_bar[cs], bytes);
                knn::bulk_g2s(c_sm + cs * kCodeBytes, a.codes + size_t(ct) * kMmaRows * QUADS, bytes, &cfull_bar[cs]);
                ++loads;
                if (++cs == uint32_t(a.code_stages)) cs = 0, parity ^= 1;
                if (++ct == a.split.cts) ct = 0;
            }
        }
    } else if (warp == kEpiWarps + 1) {
        // The whole warp goes along and one lane issues: descriptors then stay in uniform registers.  (One thread in a
        // branch of its own took 270 cycles a product, twice what the product does.)
        const uint32_t elected = elect_one();
        const uint64_t a_desc = operand_desc(smem_u32(a_sm));
        const uint64_t b_desc[2] = {operand_desc(smem_u32(b_sm)), operand_desc(smem_u32(b_sm + operand_bytes))};
        constexpr uint64_t kStep = kStepBytes >> 4;
        bool ok = true;
        for (uint32_t i = 0; i < steps && ok; ++i) {
            const uint32_t s = i & 1;
            ok = __all_sync(kFull, wait_or_abort(&full_bar[s][0], (i >> 1) & 1, i == 0 ? a.first_wait_polls : kWaitLimit, aborted) && !*aborted);
            for (int h = 0; h < 2 && ok; ++h) {
                // the half was read for the step before by the other side
                if (i) ok = __all_sync(kFull, wait_or_abort(&tempty_bar[h][s ^ 1], ((i - 1) >> 1) & 1, kWaitLimit, aborted));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem + h * 256;
                uint64_t ad = a_desc + h * ((128 * 16) >> 4), bd = b_desc[s];
                if (elected) {
#pragma unroll 4
                    for (int ks = 0; ks < split_k; ++ks, ad += kStep, bd += kStep) mma_f8(d, ad, bd, ks != 0);
                    if (h == 1) mma_commit(&empty_bar[s][0]);
                }
                if (h == 0) {
                    ok = __all_sync(kFull, wait_or_abort(&full_bar[s][1], (i >> 1) & 1, kWaitLimit, aborted));
                    if (!ok) break;
                }
                ad = a_desc + h * ((128 * 16) >> 4) + split_k * kStep, bd = b_desc[s] + split_k * kStep;
                if (elected) {
#pragma unroll 4
                    for (int ks = split_k; ks < ksteps; ++ks, ad += kStep, bd += kStep) mma_f8(d, ad, bd, true);
                    mma_commit(&tfull_bar[h][s]);
                    if (h == 1) mma_commit(&empty_bar[s][1]);
                }
            }
        }
        if (!ok) *aborted = 1;
        if (elected) mma_commit(&drain_bar);  // everything issued above has finished when this completes
    } else {
        const int quarter = warp & 3, half = (warp >> 2) & 1, side = warp >> 3;
        const uint32_t base = uint32_t(half * 128 + quarter * 32), local = base + lane;  // rows of the warp, of the lane
        const uint32_t n = uint32_t(a.n);
        const uint32_t below = (1u << lane) - 1u;
        const uint32_t addr = tmem + (uint32_t(quarter * 32) << 16) + half * 256;
        uint16_t* mine = queue[warp];
        uint4* own = reinterpret_cast<uint4*>(c_sm + size_t(a.code_stages) * kCodeBytes) + base * QUADS;  // the rows' codes
        uint32_t rt = rt0, ct = ct0, segment = 0;
        bool ok = true, begun = false;  // begun: this side has had a tile of the segment
        for (uint32_t i = 0; i < steps; ++i) {
            const uint32_t row0 = (a.tile0 + rt) * kMmaRows + base;  // the warp's first row
            const bool last = ct + 1 == a.split.cts || i + 1 == steps;  // of the segment
            if ((i & 1) == uint32_t(side)) {
                const size_t buf0 = ((size_t(blockIdx.x + rt) * kMmaRows + base) * 2 + side) * kMmaCap;
                ok = wait_or_abort(&tfull_bar[half][side], (i >> 1) & 1, kWaitLimit, aborted);
                if (__ballot_sync(kFull, !ok || *aborted)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (!begun) {
                    // the rows' other warp has to be done with the segment before, whose codes and limits are replaced
                    begun = true;
                    ok = handed_over(&finished[warp ^ 8], segment, a.handover_polls, aborted);
                    if (__ballot_sync(kFull, !ok)) {
                        ok = false;
                        break;
                    }
                    const uint32_t row = row0 + lane;
                    const bool wanted = row >= a.row_begin && row < a.row_end;
                    limit[side][local] = wanted ? int(min(a.bound[row], uint32_t(a.K))) : -1;
                    filled[side][local] = 0;
                    if (kOwnInSmem && wanted)
#pragma unroll
                        for (int w = 0; w < QUADS; ++w) own[lane * QUADS + w] = __ldg(a.codes + size_t(row) * QUADS + w);
                    __syncwarp();
                }
                const __half2 thr = dot_of_distance(a.symbols, a.K, *reinterpret_cast<volatile int*>(&limit[side][local]));
                // pairs that pass, bit j of a word: column 2 j for j < 16, else column 2 (j - 16) + 1; one load is in flight
                // while the columns of the one before are compared
                uint32_t pass[8], r[2][8];
                tmem_load16(r[0], addr);
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    tmem_wait(r[c & 1]);
                    if (c < 15) tmem_load16(r[(c + 1) & 1], addr + (c + 1) * 16);
                    uint32_t m = c & 1 ? pass[c >> 1] : 0u;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        m |= __hge2_mask(*reinterpret_cast<const __half2*>(&r[c & 1][j]), thr) & (0x00010001u << (j + (c & 1) * 8));
                    pass[c >> 1] = m;
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&tempty_bar[half][side]);

                // their exact distances, 32 pairs at a time, a lane each
                const uint32_t cs = i % uint32_t(a.code_stages);
                ok = wait_or_abort(&cfull_bar[cs], (i / uint32_t(a.code_stages)) & 1, kWaitLimit, aborted);
                if (__ballot_sync(kFull, !ok)) {
                    ok = false;
                    break;
                }
                const uint4* cand = reinterpret_cast<const uint4*>(c_sm + cs * kCodeBytes);
                const uint32_t col0 = ct * kMmaRows;
                uint32_t queued = 0;
                auto drain = [&](uint32_t m) {
                    __syncwarp();
                    queued -= m;
                    const bool act = uint32_t(lane) < m;
                    const uint32_t e = act ? mine[queued + lane] : 0u;
                    const uint32_t col = e & 255u, src = e >> 8;
                    const uint4* theirs = kOwnInSmem ? own + src * QUADS : a.codes + size_t(min(row0 + src, n - 1)) * QUADS;
                    const int d = int(code_distance<U16, QUADS>(theirs, cand + col * QUADS));
                    const uint32_t id = col0 + col;
                    if (act && id != row0 + src && d <= *reinterpret_cast<volatile int*>(&limit[side][base + src])) {
                        const size_t to = buf0 + size_t(src) * (2 * kMmaCap) + atomicAdd(&filled[side][base + src], 1u);
                        a.ids[to] = id;
                        a.dists[to] = uint8_t(d);
                    }
                    __syncwarp();
                };
                if (col0 + kMmaRows > n) {  // columns past the last node
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const uint32_t from = col0 + c * 32, have = from >= n ? 0u : (n - from < 32 ? n - from : 32u);
                        pass[c] &= ((1u << ((have + 1) / 2)) - 1u) | ((1u << (have / 2)) - 1u) << 16;
                    }
                }
                uint32_t words = 0;  // the words that have a pair left, beside the current one
#pragma unroll
                for (int c = 0; c < 8; ++c) words |= pass[c] ? 1u << c : 0u;
                uint32_t word = 0, at = 0;
                while (true) {
                    if (word == 0 && words) {
                        at = __ffs(words) - 1;
                        words &= words - 1;
                        const uint32_t w0 = at & 1 ? pass[1] : pass[0], w1 = at & 1 ? pass[3] : pass[2];
                        const uint32_t w2 = at & 1 ? pass[5] : pass[4], w3 = at & 1 ? pass[7] : pass[6];
                        const uint32_t lo = at & 2 ? w1 : w0, hi = at & 2 ? w3 : w2;
                        word = at & 4 ? hi : lo;
                    }
                    const uint32_t any = __ballot_sync(kFull, word != 0);
                    if (any == 0) break;
                    const uint32_t b = __ffs(word) - 1;
                    if (word) mine[queued + __popc(any & below)] = uint16_t(at * 32 + 2 * (b & 15) + (b >> 4) + (lane << 8));
                    word &= word - 1;
                    queued += __popc(any);
                    if (queued >= 32) drain(32);
                }
                if (queued) drain(queued);
                __syncwarp();
                if (lane == 0) mbar_arrive(&cempty_bar[cs]);

                // rows whose buffer could overflow in the next tile
                uint32_t full = __ballot_sync(kFull, filled[side][local] > kMmaKeep);
                while (full) {
                    const int src = __ffs(full) - 1;
                    full &= full - 1;
                    uint32_t count = filled[side][base + src];
                    const size_t at = buf0 + size_t(src) * (2 * kMmaCap);
                    const uint32_t T = compact_row(a.ids + at, a.dists + at, count, a.k, a.K, lane);
                    if (lane == 0) {
                        filled[side][base + src] = count;
                        // this side's later candidates have higher ids and must be strictly closer
                        atomicMin(&limit[side][base + src], int(T) - 1);
                        atomicMin(&limit[side ^ 1][base + src], int(T));
                    }
                    __syncwarp();
                }
            }
            if (last) {
                a.counts[(size_t(blockIdx.x + rt) * kMmaRows + local) * 2 + side] = begun ? filled[side][local] : 0u;
                begun = false;
                __syncwarp();
                ++segment;
                if (lane == 0) hand_over(&finished[warp], segment);
            }
            if (++ct == a.split.cts) ct = 0, ++rt;
        }
        if (!ok) *aborted = 1;
    }
    __syncthreads();
    // copies and products in flight after a lost wait end before the block's memory goes away
    if (*aborted && lane == 0) {
        if (warp == kEpiWarps) {
            atomicExch(a.status, kStatusWaitTimeout);
            for (uint32_t l = loads > 4 ? loads - 4 : 0; l < loads; ++l) mbar_wait_bounded(&full_bar[(l >> 1) & 1][l & 1], (l >> 2) & 1, kWaitLimit);
        } else if (warp == kEpiWarps + 2) {
            const uint32_t stages = uint32_t(a.code_stages);
            for (uint32_t l = loads > stages ? loads - stages : 0; l < loads; ++l) mbar_wait_bounded(&cfull_bar[l % stages], (l / stages) & 1, kWaitLimit);
        }
    }
    if (warp == kEpiWarps + 1) {
        if (lane == 0) mbar_wait_bounded(&drain_bar, 0, kWaitLimit);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
    __syncthreads();
}

// ---- results: the k best of a row's buffers by (distance, id) ---------------------------------------------------------
constexpr int kFinishWarps = 4;
constexpr int kFinishKeys = 512;

__global__ void __launch_bounds__(kFinishWarps * 32) knn_finish_kernel(KnnMmaArgs a, uint32_t rows, uint32_t* __restrict__ nbrs,
                                                                       uint16_t* __restrict__ dists, uint32_t out_row0) {
    if (a.choice.skip()) return;
    __shared__ uint64_t keys_sm[kFinishWarps][kFinishKeys];
    __shared__ uint32_t hist_sm[kFinishWarps][96];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t local = blockIdx.x * kFinishWarps + warp;
    if (local >= rows) return;
    const uint32_t row = a.tile0 * kMmaRows + local;
    if (row < a.row_begin || row >= a.row_end) return;
    uint64_t* keys = keys_sm[warp];
    uint32_t* hist = hist_sm[warp];
    const uint32_t rt = local / kMmaRows, in_tile = local % kMmaRows;
    const uint32_t seg0 = a.split.block_of(uint64_t(rt) * a.split.cts) + rt;
    const uint32_t seg1 = a.split.block_of(uint64_t(rt + 1) * a.split.cts - 1) + rt;
    // every buffer of the row, 32 entries at a time
    auto each = [&](auto&& f) {
        for (uint32_t b = seg0 * 2; b <= seg1 * 2 + 1; ++b) {
            const size_t slot = (size_t(b >> 1) * kMmaRows + in_tile) * 2 + (b & 1);
            const uint32_t count = a.counts[slot];
            for (uint32_t e = 0; e < count; e += 32) {
                const bool have = e + lane < count;
                f(have ? uint32_t(a.dists[slot * kMmaCap + e + lane]) : kFull, slot * kMmaCap + e + lane);
            }
        }
    };
    for (int i = lane; i < 96; i += 32) hist[i] = 0;
    __syncwarp();
    each([&](uint32_t d, size_t) {
        if (d != kFull) atomicAdd(hist + d, 1u);
    });
    __syncwarp();
    // T: the k-th distance (K when there are fewer); lane l owns bins 3 l .. 3 l + 2
    const uint32_t h0 = hist[3 * lane], h1 = hist[3 * lane + 1], h2 = hist[3 * lane + 2];
    uint32_t x = h0 + h1 + h2;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    const uint32_t total = __shfl_sync(kFull, x, 31), lower = x - h0 - h1 - h2;  // entries in the bins of earlier lanes
    uint32_t T = kFull, below = 0;
    if (lower < a.k && x >= a.k) {
        T = 3 * lane, below = lower;
        if (below + h0 < a.k) {
            ++T, below += h0;
            if (below + h1 < a.k) ++T, below += h1;
        }
    }
    const uint32_t owner = __ballot_sync(kFull, T != kFull);
    uint32_t last = kInvalidNode, kept = total;  // largest id of use at distance T; entries collected
    if (owner) {
        const int src = __ffs(owner) - 1;
        T = __shfl_sync(kFull, T, src);
        below = __shfl_sync(kFull, below, src);
        kept = below + hist[T];
        if (kept > uint32_t(kFinishKeys)) {  // a great many ties: the id that bounds the ones wanted
            uint32_t lo = 0, hi = kInvalidNode;
            while (lo < hi) {
                const uint32_t mid = lo + ((hi - lo) >> 1);
                uint32_t c = 0;
                each([&](uint32_t d, size_t at) { c += d == T && a.ids[at] <= mid; });
                if (__reduce_add_sync(kFull, c) >= a.k - below) hi = mid;
                else lo = mid + 1;
            }
            last = lo;
        }
    }
    uint32_t m = 0;
    each([&](uint32_t d, size_t at) {
        const uint32_t id = d <= T && d != kFull ? a.ids[at] : kInvalidNode;
        const bool take = id != kInvalidNode && (d < T || id <= last);
        const uint32_t b = __ballot_sync(kFull, take);
        if (take) keys[m + __popc(b & ((1u << lane) - 1u))] = (uint64_t(d) << 32) | id;
        m += __popc(b);
    });
    __syncwarp();
    uint32_t* out_n = nbrs + size_t(row - out_row0) * a.k;
    uint16_t* out_d = dists ? dists + size_t(row - out_row0) * a.k : nullptr;
    for (uint32_t e = lane; e < m; e += 32) {  // rank by counting: keys are distinct
        const uint64_t key = keys[e];
        uint32_t rank = 0;
#pragma unroll 4
        for (uint32_t i = 0; i < m; ++i) rank += keys[i] < key;
        if (rank < a.k) {
            out_n[rank] = uint32_t(key);
            if (out_d) out_d[rank] = uint16_t(key >> 32);
        }
    }
    for (uint32_t o = m + lane; o < a.k; o += 32) {
        out_n[o] = kInvalidNode;
        if (out_d) out_d[o] = 0xFFFF;
    }
}

template <typename CompT, int QUADS>
int launch_mma_t(cphnsw_b200_index* h, const void* d_codes, const uint32_t* padded, uint64_t n, uint32_t k, uint64_t row_begin,
                 uint64_t row_end, uint32_t* d_nbrs, uint16_t* d_dist, double most_turns, SweepChoice* other, cudaStream_t st) {
    constexpr bool U16 = sizeof(CompT) == 2;
    const CompT* codes = static_cast<const CompT*>(d_codes);
    const HashShape shape = hash_shape(int(h->K));
    const uint64_t tiles = (n + kMmaRows - 1) / kMmaRows;
    const size_t operand_bytes = size_t(shape.chunks) * kMmaRows * 16;
    const uint64_t sms = uint64_t(h->sm_count);
    // row tiles go in launches of whole waves (the buffers of a segment take 960 KB) and a last one that splits the rest
    constexpr uint64_t kWaves = 2;
    const uint64_t first_tile = row_begin / kMmaRows, end_tile = (row_end - 1) / kMmaRows + 1;
    const uint64_t most = end_tile - first_tile < kWaves * sms ? end_tile - first_tile : kWaves * sms;
    const size_t segments = size_t(most + sms);

    auto up = [](size_t b) { return (b + 255) & ~size_t(255); };
    const size_t op_b = up(size_t(tiles) * operand_bytes), hist_b = up(size_t(kBoundOrders) * kKeys * 4 + 8);
    const size_t order_b = up(size_t(kBoundOrders) * n * 4), place_b = order_b, bound_b = up(size_t(n) * 4);
    const size_t slots = segments * kMmaRows * 2;
    const size_t ids_b = up(slots * kMmaCap * 4), dists_b = up(slots * kMmaCap), counts_b = up(slots * 4);
    CPB_TRY(reserve_workspace(h, h->s_sliced, op_b + hist_b + order_b + place_b + bound_b + ids_b + dists_b + counts_b));
    unsigned char* p = h->s_sliced.as<unsigned char>();
    auto take = [&](size_t b) {
        unsigned char* r = p;
        p += b;
        return r;
    };
    uint4* operand = reinterpret_cast<uint4*>(take(op_b));
    uint32_t* hist = reinterpret_cast<uint32_t*>(take(hist_b));
    uint32_t* order = reinterpret_cast<uint32_t*>(take(order_b));
    uint32_t* place = reinterpret_cast<uint32_t*>(take(place_b));
    uint32_t* bound = reinterpret_cast<uint32_t*>(take(bound_b));

    KnnMmaArgs a;
    a.operand = operand;
    a.codes = reinterpret_cast<const uint4*>(padded);
    const size_t code_bytes = size_t(kMmaRows) * QUADS * 16, own_bytes = QUADS <= 4 ? code_bytes : 0;
    a.code_stages = 3 * operand_bytes + 4 * code_bytes + own_bytes <= kMmaSmem ? 4 : 2;  // even: a stage serves one side
    a.K = int(h->K);
    a.symbols = shape.symbols;
    a.chunks = shape.chunks;
    a.n = n;
    a.k = k;
    a.row_begin = uint32_t(row_begin);
    a.row_end = uint32_t(row_end);
    a.bound = bound;
    a.ids = reinterpret_cast<uint32_t*>(take(ids_b));
    a.dists = reinterpret_cast<uint8_t*>(take(dists_b));
    a.counts = reinterpret_cast<uint32_t*>(take(counts_b));
    a.status = h->d_status.as<uint32_t>();
    a.first_wait_polls = h->first_wait_polls;
    a.handover_polls = h->handover_polls;

    unsigned long long* load = reinterpret_cast<unsigned long long*>(hist + kBoundOrders * kKeys);
    const uint64_t rows_wanted = row_end - row_begin;
    LoadArgs sample;
    sample.groups = uint32_t((rows_wanted + 31) / 32 < kLoadGroups ? (rows_wanted + 31) / 32 : kLoadGroups);
    sample.apart = rows_wanted / sample.groups < 32 ? 32 : rows_wanted / sample.groups;
    a.choice = SweepChoice();
    if (other) {
        a.choice.load = load;
        a.choice.most = (unsigned long long)(most_turns * sample.groups * kLoadTiles);
        *other = a.choice;
        other->above = true;
    }
    CPB_CUDA(cudaMemsetAsync(hist, 0, size_t(kBoundOrders) * kKeys * 4 + 8, st));
    const dim3 by_row(unsigned((n + 255) / 256), kBoundOrders);
    key_count_kernel<CompT><<<by_row, 256, 0, st>>>(codes, n, int(h->K), hist);
    key_scan_kernel<<<kBoundOrders, 1024, 0, st>>>(hist);
    key_scatter_kernel<CompT><<<by_row, 256, 0, st>>>(codes, n, int(h->K), hist, order, place);
    auto bounds = [&](uint64_t count, uint64_t apart, const SweepChoice& choice) {
        auto go = [&](auto kernel) {
            kernel<<<unsigned((count + kBoundWarps - 1) / kBoundWarps), kBoundWarps * 32, 0, st>>>(a.codes, a.K, n, order, place, k, a.row_begin,
                                                                                                  a.row_end, bound, apart, choice);
        };
        if (QUADS > 1 && reinterpret_cast<uintptr_t>(padded) % 32 == 0) go(bound_kernel<U16, QUADS, (QUADS > 1)>);
        else go(bound_kernel<U16, QUADS, false>);
        h->launches++;
    };
    if (other) {
        bounds(uint64_t(sample.groups) * 32, sample.apart, SweepChoice());
        load_kernel<U16, QUADS><<<dim3(sample.groups, kLoadTiles), kMmaRows, 0, st>>>(a.codes, n, uint32_t(shape.symbols), uint32_t(tiles),
                                                                                     a.row_begin, a.row_end, bound, sample, load);
        h->launches++;
    }
    bounds(n, 0, a.choice);
    const uint64_t cells = tiles * shape.chunks * kMmaRows;
    expand_codes_kernel<CompT><<<unsigned((cells + 255) / 256), 256, 0, st>>>(codes, n, int(h->K), shape.symbols, shape.chunks, operand, tiles,
                                                                             a.choice);
    h->launches += 4;
    CPB_CUDA(cudaGetLastError());
    CPB_CUDA(allow_max_dynamic_smem(knn_mma_kernel<U16, QUADS>));
    for (uint64_t t0 = first_tile; t0 < end_tile;) {
        const uint64_t left = end_tile - t0;
        const uint64_t rts = left >= kWaves * sms ? kWaves * sms : (left >= sms ? left / sms * sms : left);
        a.tile0 = uint32_t(t0);
        a.split.cts = uint32_t(tiles);
        a.split.steps = rts * tiles;
        a.split.blocks = uint32_t(a.split.steps < sms ? a.split.steps : sms);
        // a block that gives up leaves its lengths unwritten; the rows it did not finish are then empty, not whatever the
        // workspace held
        CPB_CUDA(cudaMemsetAsync(a.counts, 0, size_t(a.split.blocks + rts) * kMmaRows * 2 * 4, st));
        knn_mma_kernel<U16, QUADS><<<a.split.blocks, kMmaThreads, 3 * operand_bytes + a.code_stages * code_bytes + own_bytes, st>>>(a);
        const uint32_t rows = uint32_t(rts) * kMmaRows;
        knn_finish_kernel<<<(rows + kFinishWarps - 1) / kFinishWarps, kFinishWarps * 32, 0, st>>>(a, rows, d_nbrs, d_dist, uint32_t(row_begin));
        h->launches += 2;
        CPB_CUDA(cudaGetLastError());
        t0 += rts;
    }
    return 0;
}

}  // namespace

// Plain K-component codes of up to 64 components (the operand of 256 rows has to fit shared memory three times).
bool knn_mma_supported(const cphnsw_b200_index* h) {
    return !h->binary_codes && !h->residual_bits && h->K >= 2 && hash_shape(int(h->K)).symbols != 0;
}

int launch_knn_graph_mma(cphnsw_b200_index* h, const void* d_codes, const uint32_t* padded, int words, uint64_t n, uint32_t k,
                         uint64_t row_begin, uint64_t row_end, uint32_t* d_nbrs, uint16_t* d_dist, double most_turns,
                         SweepChoice* other, cudaStream_t st) {
#define CPB_MMA(T, Q) return launch_mma_t<T, Q>(h, d_codes, padded, n, k, row_begin, row_end, d_nbrs, d_dist, most_turns, other, st)
    const bool u16 = h->comp_bytes == 2;
    switch (words) {
        case 4: if (u16) CPB_MMA(uint16_t, 1); CPB_MMA(uint8_t, 1);
        case 8: if (u16) CPB_MMA(uint16_t, 2); CPB_MMA(uint8_t, 2);
        case 16: if (u16) CPB_MMA(uint16_t, 4); CPB_MMA(uint8_t, 4);
        default: if (u16) CPB_MMA(uint16_t, 8); CPB_MMA(uint8_t, 8);
    }
#undef CPB_MMA
}

}  // namespace cpb
