// Brute-force code-distance kNN graph with the tensor cores as a filter.
//
// Same result as the two other kNN kernels (k smallest under (distance, id), self excluded).  The distance of two codes
// is K minus the number of components they share.  Every component is hashed to one of S = 8 (K <= 32) or 4 symbols and a
// symbol is written as a row of the S-point Hadamard matrix without its constant column: S - 1 values of +-1 whose dot
// product is S - 1 for equal symbols and -1 for different ones.  The dot product of two such rows of (S - 1) K values is
// S m - K, m the number of components with equal symbols, and m is at least the number of equal components: a pair whose
// dot product is below S (K - t) - K differs in more than t components.  The products run on tcgen05 in 4-bit floats with fp32
// accumulators (+-1 and integers up to 224 are exact in both), so a pair costs 2 * 256 tensor operations, at twice the rate of
// 8-bit ones, and half an instruction of the epilogue; only pairs that reach the row's threshold t have their exact distance
// computed.
//
// Row limits.  Before the sweep a bound is taken from likely neighbours: rows sorted by two of their components lie beside
// rows that share both, so windows of 32 in four such orders name groups of nodes, and once a group's rows lie together the
// k-th smallest exact distance among the 512 places beside a row bounds its final k-th distance from above.  In larger
// graphs rows that this says little about get the windows of 128 in eight orders, every row counted once.  On clustered data
// the bound is mostly right or one too high: of 100,000 x 128, K = 32, sigma 0.3, 200 rows are within it for 64 neighbours.
//
// Each pair once.  The distance is symmetric, so a tile of pairs serves the rows of both sides: row tile r meets the column
// tiles r, r + 1, .. r + half of them, cyclically, which gives every row tile the same work and every pair one product
// (where only some rows are wanted, theirs are the first tiles and the other tiles are met by all of them).  A pair passes
// at the larger of the row's limit and the largest of 32 columns', its exact distance is then held against both.  The sweep
// lists 32 rows by 32 columns where one passes; a kernel of its own compares them and keeps the rows found for a row in a
// buffer in global memory.
//
// Order.  Nodes are placed in an order in which neighbours lie together: the smallest node among the likely neighbours of a
// node names its group, followed from node to node, and within 1,024 places rows are sorted by their limit.  The pairs that
// pass are then met in a few tiles, and in all others the epilogue takes one maximum.  500k x 500k, K = 32, 64 neighbours:
// 38.8 ms with every pair twice and in the order given, 17.6 so, with 8-bit operands.  The near tiles go first: their k-th
// distances are mostly final, and limits and gates of the rest are tight.
//
// Full buffers.  Up to 32,000 nodes the sweep goes in one phase, with buffers for what the bounds let through, or, where
// clusters overlap, the near columns first.  Above, where the bounds say little, it goes by phases, every 16th (64th ..)
// column tile first, each of them as much as all before it; between them the k-th distances found are the new limits.  A
// sample of the data shows whether that is needed, and whether the filter is worth anything at all ("what the filter is
// worth" below).  A row whose buffer runs over all the same starts anew at the k-th distance of what it held, and where that
// does not do either it is compared with every node by a kernel without a buffer.
//
// Shape.  A block owns 256 rows and sweeps the column tiles of 256, a ring of whole tiles in shared memory (32 KB each at 224
// values) filled by bulk copies.  The rows' operand stays in tensor memory, so the products read only the columns' from shared
// memory.  A tile is eight units of four products, M = 128, N = 64, into seven accumulators: small units, because some 700 cycles
// lie between the issue of a unit and the reuse of its accumulator, and what is in flight has to cover them.  Two warps issue;
// sixteen read, a quarter of the columns and of either half's rows each, and hand an accumulator back as soon as it is in
// registers.  The operand is laid out by the expansion kernel in the form the tensor core reads (8-row by 16-byte core
// matrices), so a tile is one contiguous copy and no tensor map is needed.
// 500k x 500k, K = 32: the sweep takes 9.7 ms, 1,300 to 1,450 cycles a tile whose products take 1,024 (with 8-bit operands and fp16
// accumulators 15.1 ms, 2,200 of 1,792), the whole graph 14.9 against 20.4; 1M x 1M 50.9 against 72.9.  On the way, the whole graph:
// units of N = 128 and three accumulators with one warp issuing 21.0; descriptors known to be uniform and polls before waits 18.3;
// readers that hand back before they look 17.5; units of 64, a second issuing warp, columns and gates of 32 steps at a time 15.5;
// polls ahead of the products before 15.2; a step's hits listed a step later and by one atomic 14.7.  Hits
// kept in shared memory until there are five are listed by half as many atomics: 14.9 here, but 2 to 6 % less where clusters overlap.  Waits that spin instead of
// sleeping: 15.6 to 16.2.
#include <type_traits>

#include "mma_common.cuh"

namespace cpb {
namespace {

using knn::kFull;
using knn::kWaitLimit;
using knn::mbar_wait_bounded;
using knn::smem_u32;
using namespace mma;

constexpr uint32_t kMmaCap = 384;         // entries of a row's buffer, where there is more than one phase
constexpr int kMmaSlots = kMmaCap / 32;   // of them per lane
constexpr uint32_t kMmaKeep = 128;        // entries that are left of one that is cut
constexpr uint32_t kMmaFull = 256;        // entries from which on it is cut between phases
constexpr size_t kLongBuffers = size_t(128) << 20;  // bytes of the buffers of a graph of one phase, at most, if they are longer
constexpr int kBatch = 4;                 // rows compared with 32 columns at a time
constexpr uint32_t kHitRoom = 1u << 22;   // groups of 32 rows and 32 columns in the list of hits, where there are no more in all
constexpr uint32_t kStepHits = 64;        // such groups in a step
constexpr uint32_t kSection = 8192, kSections = 672;  // else: entries of a section of the list, and sections (63 MB in all)
constexpr uint32_t kDrain = 2048;         // hits of a section that its block compares itself, at a time, when there are no others
constexpr uint32_t kLeastRoom = 512;      // room that a section has to have for its block to go on with it
static_assert(kLeastRoom >= kStepHits && kSection - kLeastRoom >= kDrain, "a section has room for a step, or hits to compare");
constexpr uint64_t kLaunchSteps = 1u << 22;
constexpr uint32_t kCheckBlocks = 4;      // blocks of the check an SM
constexpr uint32_t kNearColumns = 8, kNearFrom = 64;  // column tiles that are swept first, of so many at least
constexpr int kEpiWarps = 16;             // epilogue warps: a quarter of the lanes and of the columns, of both halves of the rows
constexpr int kMmaWarps = 2;              // warps that issue products, see there
constexpr int kMmaThreads = (kEpiWarps + 1 + kMmaWarps) * 32;  // and one for the operands' copies
constexpr int kMaxStages = 8;             // of a tile each
constexpr size_t kMmaSmem = 216 * 1024;   // dynamic shared memory a block may use beside its 3 KB of static
constexpr int kSortRows = 1024;           // places sorted by limit together
constexpr uint32_t kFirstColumns = 8;      // column tiles of the first phase, at most
constexpr uint32_t kOnePhase = 64;         // up to so many (32,000 nodes) there is one, or the near columns and the rest, and calm
                                           // data have no second bounds: what these would save costs less than their launches
                                           // (16,000 x 128, sigma 0.3: 525 us with phases and second bounds, 392 without)
constexpr uint32_t kOnePhaseBounds = 48;   // from here on (24,600 nodes) data that are not calm get the second bounds all the same
                                           // (300-d, two bytes, sigma 0.6: 30,000 5,994 us without, 4,056 with; K = 64, sigma 0.5,
                                           // 20,000: 1,662 and 1,881)
constexpr int kBoundOrders = 8;           // orders of likely neighbours
constexpr int kBoundWindow = 128;         // rows looked at per order
constexpr int kNameOrders = 4, kNameWindow = 32;  // of them for the names of the groups
constexpr uint64_t kOrderNodes = 4096;    // fewer are met in the order given (5,000 x 128: 225 us so, 210 in groups)
constexpr uint32_t kKeys = 65536;

// symbols and values of a code shape; 0 symbols: not served
struct HashShape {
    int symbols, chunks;  // chunks: 16-byte pieces of a row's operand, 32 values each, an even number
};
__host__ __device__ inline HashShape hash_shape(int K) {
    HashShape s;
    s.symbols = K <= 32 ? 8 : (K <= 64 ? 4 : 0);
    const int values = K * (s.symbols - 1);
    s.chunks = (values + 63) / 64 * 2;
    return s;
}

__device__ __forceinline__ uint32_t symbol_of(uint32_t comp, uint32_t symbols) {
    return (comp ^ (comp >> 3) ^ (comp >> 6) ^ (comp >> 9)) & (symbols - 1);
}

// ---- operand: [tile of 256 rows][chunk][row][32 values of 4 bits] ---------------------------------------------------
// codes: padded rows of `stride` components in their places
template <typename CompT>
__global__ void expand_codes_kernel(const CompT* __restrict__ codes, int stride, const uint2* __restrict__ place, int K, int symbols,
                                    int chunks, uint4* __restrict__ out, uint64_t tiles, SweepChoice choice) {
    if (choice.skip()) return;
    const uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= tiles * chunks * kMmaRows) return;
    const int r = int(t % kMmaRows), c = int(t / kMmaRows % chunks);
    const uint64_t row = t / (uint64_t(kMmaRows) * chunks) * kMmaRows + r;
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (place[row].x != kInvalidNode) {
        const CompT* code = codes + row * stride;
        int comp = c * 32 / (symbols - 1), j = c * 32 % (symbols - 1) + 1;
        uint32_t h = comp < K ? symbol_of(code[comp], uint32_t(symbols)) : 0u;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const uint32_t e2m1 = (__popc(h & uint32_t(j)) & 1) ? 0xAu : 0x2u;  // -1 : +1
            if (comp < K) w[i / 8] |= e2m1 << (4 * (i % 8));
            if (++j == symbols) {
                j = 1;
                ++comp;
                if (comp < K) h = symbol_of(code[comp], uint32_t(symbols));
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

// What the sample counts: turns, and the pairs that are truly within the rows' bounds.  Up to kCalmEntries of them a row
// the buffers hold what the whole sweep finds, and up to kCalmTurns there is little to gain from limits that fall on the
// way: it then goes in one phase (400k x 128, mixture sigma 0.5, 29 turns: 185 ms in one, 143 in seven).  Graphs of one phase
// take the near columns by themselves from kSmallCalm turns in all on, where the launches around them, 60 us, are made up for:
// K = 32, sigma 0.6, 20,000 x 128 (77 turns) 1,256 us in one, 1,177 so, 10,000 (106) 544 and 591; in 64-byte codes from
// 0.56 of that (300-d, two bytes, 30,000, 151 turns: 7,982 and 4,056; 14,000, 61 turns: 921 and 951).
struct LoadCounts {
    unsigned long long turns;
    uint32_t within;
};
constexpr double kCalmEntries = 230, kCalmTurns = 20, kSmallCalm = 25e9;
struct Calm {
    const LoadCounts* counts = nullptr;  // (nullptr: not known)
    uint32_t most = 0;
    unsigned long long most_turns = 0;
    __device__ __forceinline__ bool yes() const { return counts && counts->within <= most && counts->turns <= most_turns; }
};

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
constexpr uint32_t kCloseRows = 12;
template <bool U16, int QUADS, bool SECTORS, int ORDERS, int WINDOW>
__global__ void __launch_bounds__(kBoundWarps * 32)
bound_kernel(const uint4* __restrict__ codes, int K, uint64_t n, const uint32_t* __restrict__ order, const uint32_t* __restrict__ place,
             uint32_t k, uint32_t row_begin, uint32_t row_end, uint32_t* __restrict__ bound, uint32_t* __restrict__ group, uint32_t* __restrict__ mate,
             uint64_t apart /* of LoadArgs: its rows only; 0: all rows */, const uint32_t* __restrict__ listed /* only these rows */,
             const uint32_t* __restrict__ listed_count, SweepChoice choice, Calm calm) {
    if (choice.skip() || calm.yes()) return;
    constexpr int S = WINDOW / 32, N = ORDERS * S;
    constexpr uint32_t kSeenSlots = N * 32 > 512 ? 1024 : 512;
    __shared__ uint32_t seen_sm[kBoundWarps][kSeenSlots];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t warps = uint64_t(gridDim.x) * kBoundWarps, many = listed ? *listed_count : apart ? warps : n;
    for (uint64_t at = uint64_t(blockIdx.x) * kBoundWarps + warp; at < many; at += warps) {
        const uint64_t wanted = listed ? listed[at] : apart ? row_begin + at / 32 * apart + at % 32 : order[at];
        if (wanted < row_begin || wanted >= row_end) continue;
        const uint32_t row = uint32_t(wanted);
        uint32_t* seen = seen_sm[warp];
        for (uint32_t i = lane; i < kSeenSlots / 4; i += 32) reinterpret_cast<uint4*>(seen)[i] = make_uint4(kFull, kFull, kFull, kFull);
        const uint32_t where = lane < ORDERS ? place[uint64_t(row) * kBoundOrders + lane] : 0u;
        uint32_t id[N], dist[N / 4] = {};  // distances a byte each
        uint4 own[QUADS];
#pragma unroll
        for (int w = 0; w < QUADS; ++w) own[w] = __ldg(codes + size_t(row) * QUADS + w);
#pragma unroll
        for (int o = 0; o < ORDERS; ++o) {
            const uint64_t pos = __shfl_sync(kFull, where, o);
            uint64_t first = pos < WINDOW / 2 ? 0 : pos - WINDOW / 2;
            if (first + WINDOW > n) first = n > WINDOW ? n - WINDOW : 0;
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
                uint32_t slot = (id[i] * 0x9E3779B1u) >> (kSeenSlots == 1024 ? 22 : 23);
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
        if (listed) {
            if (lane == 0 && T < bound[row]) bound[row] = T;
            __syncwarp();
            continue;
        }
        // of the closest few, as far as they are likely in its cluster, the smallest wanted node names the row's group, the
        // largest is a mate
        const uint32_t close = min(kth_packed(dist, kCloseRows, K), uint32_t(K) * 5 / 8);
        uint32_t least = row, most = row;
#pragma unroll
        for (int i = 0; i < N; ++i)
            if ((dist[i / 4] >> (8 * (i % 4)) & 127u) <= close && id[i] >= row_begin && id[i] < row_end) least = min(least, id[i]), most = max(most, id[i]);
        least = __reduce_min_sync(kFull, least);
        most = __reduce_max_sync(kFull, most);
        if (lane == 0) bound[row] = T, group[row] = least, mate[row] = most;
        __syncwarp();
    }
}

// Bounds from the rows that lie beside a row once its group lies together: 32 rows a block, the 512 places around them from
// shared memory, a quarter of them for each warp, the k-th smallest of a row's distances.  (The windows of the orders alone,
// eight of 128 for every row, took 8.3 us per 1,000 rows, gathers through the L1; the windows of four of 32 for the names of
// the groups take 1.2, the order 0.7 and this 1.2.)
constexpr int kBesideRows = 32, kBesideWarps = 4, kBesidePlaces = 512;
template <bool U16, int QUADS>
__global__ void __launch_bounds__(kBesideWarps * 32) beside_kernel(const uint4* __restrict__ codes, const uint32_t* __restrict__ grouped, uint32_t rows,
                                                                   int K, uint32_t k, uint32_t* __restrict__ bound,
                                                                   uint32_t* __restrict__ far, uint32_t* __restrict__ far_count, SweepChoice choice) {
    if (choice.skip()) return;
    extern __shared__ __align__(16) unsigned char beside_smem[];
    uint4* code = reinterpret_cast<uint4*>(beside_smem);                                   // [kBesidePlaces][QUADS]
    uint16_t* count = reinterpret_cast<uint16_t*>(code + kBesidePlaces * QUADS);           // [distance][warp][row]
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, row0 = blockIdx.x * kBesideRows, own_place = row0 + lane;
    const uint32_t ahead = (kBesidePlaces - kBesideRows) / 2;
    uint32_t from = row0 < ahead ? 0 : row0 - ahead;
    if (from + kBesidePlaces > rows) from = rows > uint32_t(kBesidePlaces) ? rows - kBesidePlaces : 0;
    const uint32_t have = min(rows - from, uint32_t(kBesidePlaces));
    for (uint32_t i = tid; i < have * QUADS; i += kBesideWarps * 32) code[i] = __ldg(codes + size_t(grouped[from + i / QUADS]) * QUADS + i % QUADS);
    for (int d = 0; d <= K; ++d) count[d * kBesideWarps * 32 + tid] = 0;
    __syncthreads();
    uint4 own[QUADS];
#pragma unroll
    for (int w = 0; w < QUADS; ++w) own[w] = code[min(own_place, rows - 1) * QUADS - from * QUADS + w];
    const uint32_t j1 = min(have, (warp + 1) * (kBesidePlaces / kBesideWarps));
#pragma unroll 4
    for (uint32_t j = warp * (kBesidePlaces / kBesideWarps); j < j1; ++j) {
        const uint32_t d = code_distance<U16, QUADS>(own, code + j * QUADS);
        count[d * kBesideWarps * 32 + tid] += from + j != own_place;
    }
    __syncthreads();
    if (warp != 0 || own_place >= rows) return;
    const uint32_t node = grouped[own_place], before = bound[node];
    uint32_t T = 0, upto = 0;
    for (; T < uint32_t(K); ++T) {
        for (int w = 0; w < kBesideWarps; ++w) upto += count[(T * kBesideWarps + w) * 32 + lane];
        if (upto >= k) break;
    }
    if (T < before) bound[node] = T;
    if (min(T, before) > uint32_t(K) * 5 / 8) far[atomicAdd(far_count, 1u)] = node;
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
                                                        LoadCounts* load) {
    __shared__ uint4 rows_sm[32][QUADS], plain_sm[32][QUADS];
    __shared__ uint32_t bound_sm[32], passed[32], within;
    const uint32_t g = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const uint64_t row0 = row_begin + g * a.apart;
    const uint32_t have = uint32_t(row_end - row0 < 32 ? row_end - row0 : 32);
    const uint32_t tile = uint32_t((uint64_t(blockIdx.y) * a.groups + g) * tiles / (uint64_t(a.groups) * kLoadTiles));
    auto hashed = [&](uint4 v) {
        return make_uint4(symbols_of<U16>(v.x, symbols), symbols_of<U16>(v.y, symbols), symbols_of<U16>(v.z, symbols), symbols_of<U16>(v.w, symbols));
    };
    for (uint32_t i = tid; i < have * QUADS; i += kMmaRows) {
        const uint4 v = __ldg(codes + row0 * QUADS + i);
        plain_sm[i / QUADS][i % QUADS] = v;
        rows_sm[i / QUADS][i % QUADS] = hashed(v);
    }
    if (tid < 32) passed[tid] = 0, bound_sm[tid] = tid < have ? bound[row0 + tid] : 0u;
    if (tid == 0) within = 0;
    const uint64_t col = uint64_t(tile) * kMmaRows + tid;
    uint4 plain[QUADS], own[QUADS];
#pragma unroll
    for (int w = 0; w < QUADS; ++w) plain[w] = __ldg(codes + (col < n ? col : 0) * QUADS + w), own[w] = hashed(plain[w]);
    __syncthreads();
    uint32_t near = 0;
    for (uint32_t r = 0; r < have; ++r) {
        const bool pass = col < n && code_distance<U16, QUADS>(rows_sm[r], own) <= bound_sm[r];
        const uint32_t m = __ballot_sync(kFull, pass);
        if (lane == 0 && m) atomicAdd(&passed[r], __popc(m));
        if (pass) near += code_distance<U16, QUADS>(plain_sm[r], plain) <= bound_sm[r];
    }
    if (near) atomicAdd(&within, near);
    __syncthreads();
    if (tid < 32) {
        const uint32_t most = __reduce_max_sync(kFull, passed[tid]), all = __reduce_add_sync(kFull, passed[tid]);
        if (tid == 0) {
            atomicAdd(&load->turns, (unsigned long long)(most + (all + 31) / 32));
            atomicAdd(&load->within, within);
        }
    }
}

// ---- tcgen05 pieces ------------------------------------------------------------------------------------------------
// D fp32, A and B e2m1 with a scale of ue8m0 for every 32 values, both K-major, M = 128, N = 64.  Tensor memory: accumulators
// of 64 columns each, and the block's rows, a half of them in 32 columns, 8 values a word.  The scales, all of them one, lie in
// the last four columns of the halves, for A in the first and for B in the second: where a row has as many values these columns
// meet zeros of the other operand (28 to 32 components of 7 values are 196 to 224 of 256).
constexpr uint32_t kUnitCols = 64, kUnits = 7, kUnitsStep = 8;  // columns of an accumulator; accumulators; units of a step
constexpr uint32_t kRowsAt = kUnits * kUnitCols, kRowsCols = 32, kScaleCols = 4;
constexpr uint32_t kScalesAt = kRowsAt + kRowsCols - kScaleCols;
constexpr uint32_t kScaleOne = 0x7f7f7f7fu;
static_assert(kRowsAt + 2 * kRowsCols == kTmemCols, "tensor memory");
constexpr uint32_t kIdesc = (1u << 7) | (1u << 10) | ((kUnitCols >> 3) << 17) | (1u << 23) | (uint32_t(128 >> 7) << 27);

__device__ __forceinline__ void mma_f4(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t scales, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], %2, %3, [%4], [%5], p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b), "r"(kIdesc), "r"(scales), "r"(scales + kRowsCols), "r"(uint32_t(accumulate))
        : "memory");
}
// 32 columns of the warp's 32 lanes of tensor memory: asked for, and waited for
__device__ __forceinline__ void tmem_load32(uint32_t (&r)[32], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, "
        "%21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(addr)
        : "memory");
}
// (the registers are operands so that no use of them moves in front of the wait)
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[32], uint32_t (&q)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(r[i]), "+r"(q[i]));
}
__device__ __forceinline__ void tmem_store4(uint32_t addr, const uint4& v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ int largest(const uint32_t (&v)[32]) {
    int m[12];
#pragma unroll
    for (int i = 0; i < 10; ++i) m[i] = __vimax3_s32(int(v[3 * i]), int(v[3 * i + 1]), int(v[3 * i + 2]));
    m[10] = int(v[30]), m[11] = int(v[31]);
#pragma unroll
    for (int i = 0; i < 4; ++i) m[i] = __vimax3_s32(m[3 * i], m[3 * i + 1], m[3 * i + 2]);
    return __vimax3_s32(m[0], m[1], max(m[2], m[3]));
}

// ---- which tiles meet ------------------------------------------------------------------------------------------------
// The first row_tiles tiles hold the rows wanted.  Row tile r meets the tiles r + j, j <= row_tiles / 2, of them, cyclically
// (for an even number the farthest pair is met from both sides, each for its own rows), and all tiles behind them.
struct Meet {
    uint32_t tiles, row_tiles;
    __host__ __device__ uint32_t columns() const { return row_tiles / 2 + 1 + (tiles - row_tiles); }
    __device__ uint32_t column(uint32_t rt, uint32_t j) const {
        if (j > row_tiles / 2) return row_tiles + (j - row_tiles / 2 - 1);
        const uint32_t ct = rt + j;
        return ct >= row_tiles ? ct - row_tiles : ct;
    }
    // the column's rows take part with limits of their own
    __device__ bool both(uint32_t rt, uint32_t ct) const {
        const uint32_t j = ct >= rt ? ct - rt : ct + row_tiles - rt;
        return ct < row_tiles && j != 0 && 2 * j != row_tiles;
    }
};
// The columns of one launch: from `base` on every stride-th, or the odd ones of those; `count` of them from the from-th on.
struct Phase {
    uint32_t base, stride;
    bool odd;
    uint32_t from, count;
    __host__ __device__ uint32_t columns(uint32_t of) const {  // in all
        const uint32_t c = (of - base + stride - 1) / stride;
        return odd ? c / 2 : c;
    }
    __device__ uint32_t column(uint32_t i) const { return base + stride * (odd ? 2 * (from + i) + 1 : from + i); }
};
// What a block does: whole row tiles, a grid's width apart, so that the blocks meet the same column tiles at about the same
// time and a tile comes from L2; then its part of the steps of the row tiles left over.
struct Walk {
    uint32_t len, whole, rt, at;  // steps of a row tile; whole row tiles to come; row tile and step
    uint32_t col;                 // the step's column (at, or at * hop % len)
    uint32_t steps, apart;        // of the block; rows between its whole row tiles
    uint32_t rest_rt, rest_at;    // where its part of the rest begins
    uint32_t hop;                 // the rest goes round a row tile's columns by this many: neighbouring columns are far apart
    __device__ Walk(uint32_t row_tiles, uint32_t len_) {
        const uint32_t blocks = gridDim.x, b = blockIdx.x;
        len = len_;
        apart = blocks;
        whole = row_tiles / blocks;
        const uint64_t rest = uint64_t(row_tiles % blocks) * len, r0 = b * rest / blocks, r1 = (b + 1) * rest / blocks;
        rest_rt = whole * blocks + uint32_t(r0 / len), rest_at = uint32_t(r0 % len);
        steps = whole * len + uint32_t(r1 - r0);
        rt = whole ? b : rest_rt;
        at = whole ? 0 : rest_at;
        // in time, some 0.618 of the way round (hop is the inverse of that number without a common divisor with len)
        hop = 1;
        if (whole * blocks < row_tiles && len > 2) {
            for (int apart_in_time = int(0.618f * float(len));; ++apart_in_time) {
                int r0 = int(len), r1 = apart_in_time, t0 = 0, t1 = 1;
                while (r1) {
                    const int q = r0 / r1, r = r0 - q * r1, t = t0 - q * t1;
                    r0 = r1, r1 = r, t0 = t1, t1 = t;
                }
                if (r0 == 1) {
                    hop = uint32_t(t0 < 0 ? t0 + int(len) : t0);
                    break;
                }
            }
        }
        col = column(0);
    }
    __device__ void next() {
        if (++at < len) {
            col += whole ? 1 : hop;
            if (col >= len) col -= len;
        } else {
            next_rows();
        }
    }
    // by row tiles: the steps until it changes, their columns, and the change
    __device__ uint32_t run() const { return len - at; }
    __device__ uint32_t column(uint32_t ahead) const { return whole ? at + ahead : uint32_t(uint64_t(at + ahead) * hop % len); }
    __device__ void next_rows() {
        at = 0;
        if (whole && --whole) rt += apart;
        else if (whole == 0 && rt >= rest_rt) ++rt;
        else rt = rest_rt, at = rest_at;
        col = column(0);
    }
};

struct KnnMmaArgs {
    const uint4* operand;   // [tiles][chunks][256], places in order
    const uint4* codes;     // [tiles * 256] padded rows, places in order
    uint2* place;           // [tiles * 256] the node at a place (kInvalidNode: none), largest distance of use to it (-1: none)
    int16_t* gate;          // [row_tiles][8] what a product reaches at the largest limit of 32 places (gate_of)
    int K, symbols, chunks, stages;
    uint32_t k;
    Meet meet;
    Phase phase;
    enum { kAlways, kAllIfCalm, kNotIfCalm } when;  // calm data: the second takes all its columns at once, the third has nothing to do
    bool wide;              // entries of two words
    uint32_t cap;           // entries of a row's buffer: kMmaCap, or more (of one word each) in a graph of one phase
    uint32_t* entries;      // [row_tiles * 256][cap]
    uint32_t* counts;       // [row_tiles * 256] entries; above cap: some were lost
    // 32 rows and 32 columns among which a product reaches its gate, in one list or in sections
    uint4* hits;             // first row, first column, rows, both
    uint32_t* hit_count;
    uint2* places;           // [kSections][kSection] first row | both, first column
    uint32_t* rows;          // [kSections][kSection]
    uint32_t* section_hits;  // [kSections]
    uint32_t* taken;         // sections that blocks have taken behind their first ones, of which there is one a block
    uint32_t blocks;         // of the sweep
    uint32_t* status;
    uint32_t first_wait_polls, handover_polls;
    SweepChoice choice;
    Calm calm;
};

// The dot product a pair at distance <= t reaches at least, as the upper half of its float's bits (the lower is zero, dot
// products are 224 at most): above zero floats compare as their bits do, and those below zero are below; where zero or less
// is enough every product will do.  t < 0: none does.
__device__ __forceinline__ int gate_of(int symbols, int K, int t) {
    const int dot = symbols * (K - t) - K;
    return t < 0 ? 0x7fff : (dot > 0 ? int(__float_as_uint(float(dot)) >> 16) : -0x8000);
}

// The entries of a row's buffer: (distance, node), packed in a word up to kPackedNodes nodes, in two above.
constexpr uint32_t kPackedNodes = 1u << 25;
struct Entry {
    uint32_t d, node;
};
__device__ __forceinline__ Entry load_entry(const uint32_t* buf, bool wide, uint32_t e) {
    if (wide) {
        const uint2 v = reinterpret_cast<const uint2*>(buf)[e];
        return Entry{v.x, v.y};
    }
    const uint32_t v = buf[e];
    return Entry{v >> 25, v & (kPackedNodes - 1u)};
}
__device__ __forceinline__ void store_entry(uint32_t* buf, bool wide, uint32_t e, uint32_t d, uint32_t node) {
    if (wide) reinterpret_cast<uint2*>(buf)[e] = make_uint2(d, node);
    else buf[e] = d << 25 | node;
}
__device__ __forceinline__ uint32_t* buffer_of(const KnnMmaArgs& a, uint32_t place) {
    return a.entries + size_t(place) * (a.cap * (a.wide ? 2 : 1));
}

// What is nearer than T, and at T up to node `last`, moves to the front of the buffer; returns their number.  By the whole warp.
__device__ __forceinline__ uint32_t keep_entries(uint32_t* buf, bool wide, uint32_t count, uint32_t T, uint32_t last, int lane) {
    __syncwarp();
    uint32_t at = 0;
#pragma unroll 1
    for (uint32_t e = lane; e < (count + 31u) / 32 * 32; e += 32) {  // (an entry moves down or stays)
        const Entry x = e < count ? load_entry(buf, wide, e) : Entry{kFull, kInvalidNode};
        const bool keep = x.d < T || (x.d == T && x.node <= last);
        const uint32_t m = __ballot_sync(kFull, keep);
        __syncwarp();
        if (keep) store_entry(buf, wide, at + __popc(m & ((1u << lane) - 1u)), x.d, x.node);
        at += __popc(m);
        __syncwarp();
    }
    return at;
}

// The row's buffer shrinks to its k best (or all that are no worse than the k-th, up to kMmaKeep).  By the whole warp;
// returns the k-th distance and the new count.
__device__ __forceinline__ uint32_t compact_row(uint32_t* buf, bool wide, uint32_t& count, uint32_t k, int K, int lane) {
    uint32_t dist[kMmaSlots];
#pragma unroll
    for (int s = 0; s < kMmaSlots; ++s) {
        const uint32_t e = uint32_t(s * 32 + lane);
        dist[s] = e < count ? load_entry(buf, wide, e).d : kFull;
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
            for (uint32_t e = lane; e < count; e += 32) {
                const Entry x = load_entry(buf, wide, e);
                c += x.d == T && x.node <= mid;
            }
            if (__reduce_add_sync(kFull, c) >= k - below) hi = mid;
            else lo = mid + 1;
        }
        last = lo;
    }
    count = keep_entries(buf, wide, count, T, last, lane);
    return T;
}

// The exact distances of `rows` of the 32 places from row0 on to the 32 from col0 on, a column per lane and kBatch rows at a
// time, and the rows found to the buffers they are of use to.  By the whole warp; row: the lane's place among the rows.
template <bool U16, int QUADS>
__device__ __forceinline__ void compare_rows(const KnnMmaArgs& a, uint32_t rows, uint32_t row0, uint2 row, uint32_t col0, bool both, int lane) {
    if (rows == 0) return;
    const uint32_t below = (1u << lane) - 1u, col = col0 + lane;
    const uint2 p = __ldg(a.place + col);
    uint4 own[QUADS];  // the lane's column
#pragma unroll
    for (int w = 0; w < QUADS; ++w) own[w] = __ldg(a.codes + size_t(col) * QUADS + w);
    while (rows) {
        uint32_t src[kBatch], here[kBatch], dist = 0, there = 0;  // columns of use to a row; rows of use to the column
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
            src[b] = here[b] = 0;
            if (rows) {
                src[b] = __ffs(rows) - 1;
                rows &= rows - 1;
                uint4 theirs[QUADS];
#pragma unroll
                for (int w = 0; w < QUADS; ++w) theirs[w] = __ldg(a.codes + size_t(row0 + src[b]) * QUADS + w);
                const uint32_t d = code_distance<U16, QUADS>(own, theirs);
                const int row_limit = int(__shfl_sync(kFull, row.y, src[b]));
                const uint32_t row_node = __shfl_sync(kFull, row.x, src[b]);
                dist |= d << (8 * b);
                here[b] = __ballot_sync(kFull, int(d) <= row_limit && p.x != kInvalidNode && col != row0 + src[b]);
                there |= both && int(d) <= int(p.y) && row_node != kInvalidNode ? 1u << b : 0u;
            }
        }
        uint32_t slot = 0, at = 0;
#pragma unroll
        for (int b = 0; b < kBatch; ++b)
            if (here[b] && uint32_t(lane) == src[b]) slot = atomicAdd(a.counts + row0 + lane, uint32_t(__popc(here[b])));
        if (there) at = atomicAdd(a.counts + col, uint32_t(__popc(there)));
        __syncwarp();
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
            const uint32_t d = dist >> (8 * b) & 255u;
            const uint32_t to = __shfl_sync(kFull, slot, src[b]) + __popc(here[b] & below);
            const uint32_t row_node = __shfl_sync(kFull, row.x, src[b]);
            if ((here[b] >> lane & 1u) && to < a.cap) store_entry(buffer_of(a, row0 + src[b]), a.wide, to, d, p.x);
            if (there >> b & 1u) {
                if (at < a.cap) store_entry(buffer_of(a, col), a.wide, at, d, row_node);
                ++at;
            }
        }
        __syncwarp();
    }
}

struct SectionHits {
    uint32_t of[kSections], upto[kSections], groups[kSections / 32];  // hits of a section; of its group of 32 up to it; up to a group
};
// The place of the e-th hit.  (A call, and the kernel has the registers that comparing takes and no more.)
__device__ __noinline__ uint32_t place_of_hit(const SectionHits& hits, uint32_t e) {
    const int lane = threadIdx.x & 31;
    constexpr int kGroups = int(kSections / 32);
    const int g = __popc(__ballot_sync(kFull, lane < kGroups && hits.groups[min(lane, kGroups - 1)] <= e));
    const uint32_t in_group = e - (g ? hits.groups[g - 1] : 0u);
    const int s = __popc(__ballot_sync(kFull, hits.upto[32 * g + lane] <= in_group));
    return uint32_t(32 * g + s) * kSection + in_group - (s ? hits.upto[32 * g + s - 1] : 0u);
}

// What the sweep has listed.  What bounds it is latency, of the rows and of the places in the buffers, some 1,500 cycles a
// batch, and from 64 bytes on the comparing: 32 warps an SM, of 128 bytes 16 with registers enough for a batch in flight
// (60,000 x 300, two bytes, K = 64: 24.9 ms with 24 warps, 23.6 so).  (In the sweep's own epilogue, two warps a scheduler, the
// products wait for it: 100k x 128 clustered 3.2 ms in all, 2.1 with the list.)
constexpr int kCheckWarps = 8;
template <bool U16, int QUADS>
__global__ void __launch_bounds__(kCheckWarps * 32, (QUADS > 4 ? 2 : 0)) knn_check_kernel(KnnMmaArgs a) {
    if (a.choice.skip() || (a.when == KnnMmaArgs::kNotIfCalm && a.calm.yes())) return;
    const int lane = threadIdx.x & 31;
    const uint32_t warp = blockIdx.x * kCheckWarps + (threadIdx.x >> 5), warps = gridDim.x * kCheckWarps;
    const uint32_t many = *a.hit_count;
    const uint32_t parts = many < 8 * warps ? 4 : 1;  // few: eight rows a warp
    for (uint32_t i = warp; i < many * parts; i += warps) {
        const uint4 h = __ldg(a.hits + i / parts);
        const uint32_t rows = parts == 1 ? h.z : h.z & (0xffu << (8 * (i % parts)));
        compare_rows<U16, QUADS>(a, rows, h.x, __ldg(a.place + h.x + lane), h.y, h.w != 0, lane);
    }
}
template <bool U16, int QUADS>
__device__ __forceinline__ void compare_hit(const KnnMmaArgs& a, uint2 at, uint32_t rows, int lane) {
    const uint32_t row0 = at.x & ~31u;
    compare_rows<U16, QUADS>(a, rows, row0, __ldg(a.place + row0 + lane), at.y, at.x & 1u, lane);
}

// The same for hits in sections: few are taken one by one, many place by place, those behind a section's hits too, which costs less
// than to look for each.
template <bool U16, int QUADS>
__global__ void __launch_bounds__(kCheckWarps * 32, (QUADS > 4 ? 2 : 0)) knn_check_sections_kernel(KnnMmaArgs a) {
    if (a.choice.skip() || (a.when == KnnMmaArgs::kNotIfCalm && a.calm.yes())) return;
    const int lane = threadIdx.x & 31;
    const uint32_t warp = blockIdx.x * kCheckWarps + (threadIdx.x >> 5), warps = gridDim.x * kCheckWarps;
    constexpr int kGroups = int(kSections / 32);
    __shared__ SectionHits hits;
    const uint32_t used = min(a.blocks + *a.taken, kSections);
    auto scan = [&](uint32_t x) {  // inclusive, over the lanes
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, x, d);
            if (lane >= d) x += y;
        }
        return x;
    };
#pragma unroll
    for (int g = int(threadIdx.x >> 5); g < kGroups; g += kCheckWarps) {
        const uint32_t s = uint32_t(32 * g + lane), own = s < used ? __ldg(a.section_hits + s) : 0u, x = scan(own);
        hits.of[s] = own, hits.upto[s] = x;
        if (lane == 31) hits.groups[g] = x;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint32_t x = scan(lane < kGroups ? hits.groups[lane] : 0u);
        if (lane < kGroups) hits.groups[lane] = x;
    }
    __syncthreads();
    const uint32_t many = hits.groups[kGroups - 1];
    if (many >= 64 * warps && many > used * (kSection / 4)) {
        for (uint32_t at = warp; at < used * kSection; at += warps)
            if (at % kSection < hits.of[at / kSection]) compare_hit<U16, QUADS>(a, __ldg(a.places + at), __ldg(a.rows + at), lane);
        return;
    }
    const uint32_t parts = many < 8 * warps ? 4 : 1;  // few: eight rows a warp
    for (uint32_t i = warp; i < many * parts; i += warps) {
        const uint32_t at = place_of_hit(hits, i / parts), rows = __ldg(a.rows + at);
        compare_hit<U16, QUADS>(a, __ldg(a.places + at), parts == 1 ? rows : rows & (0xffu << (8 * (i % parts))), lane);
    }
}

__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// The products of a block's steps, KSTEPS of 64 values of K each, by two warps: the first has the even units and four of the
// accumulators, the second the odd units and three.  (A warp only waits for units of its own: the other's barriers could be two
// phases on.)  The whole warp goes along and one lane issues: descriptors then stay in uniform registers.  (One thread in a
// branch of its own took 270 cycles a product, which takes 32.)  A unit of four products takes 128 cycles, so what lies between
// them counts: a wait that is over is one poll and a vote.
template <int KSTEPS>
__device__ __forceinline__ bool issue_products(const KnnMmaArgs& a, Walk walk, uint32_t steps, uint32_t first, uint32_t tmem, uint32_t smem,
                                               uint32_t operand_bytes, uint32_t elected, uint64_t* full_bar, uint64_t* empty_bar, uint64_t* tfull_bar,
                                               uint64_t* tempty_bar, uint64_t* rows_bar, uint64_t* done_bar, volatile int* aborted) {
    auto wait = [&](bool over, uint64_t* bar, uint32_t parity, uint32_t limit) {
        return __all_sync(kFull, over) || __all_sync(kFull, wait_or_abort(bar, parity, limit, aborted));
    };
    // the unit that had the accumulator of unit 2 v + first of step i was read: the same of the step before, or the second warp's
    // third before
    auto emptied = [&](uint32_t v, uint32_t i, uint64_t*& bar, uint32_t& parity) {
        bar = &tempty_bar[first ? (v == 3 ? 1 : 2 * v + 3) : 2 * v];
        parity = (first && v == 3 ? i : i + 1) & 1;
    };
    constexpr uint64_t kStep = (2 * kMmaRows * 16) >> 4;  // two 16-byte chunks of 256 rows
    const uint64_t b_desc = operand_desc(smem);
    const uint32_t stages = uint32_t(a.stages);
    uint32_t stage = 0, parity = 0, rows_parity = 0, turn = 0;  // turn: among the second warp's accumulators
    uint32_t left = walk.run();
    bool fresh = true;  // of a new row tile
    bool full = false, empty = true;  // what the polls said (a step's first waits, of a barrier that nothing has used, are over)
    uint64_t* bar;
    uint32_t of;
    for (uint32_t i = 0; i < steps; ++i) {
        if (!wait(full, &full_bar[stage], parity, i == 0 ? a.first_wait_polls : kWaitLimit)) return false;
        if (fresh) {
            if (!wait(false, rows_bar, rows_parity, kWaitLimit)) return false;
            rows_parity ^= 1;
        }
        fresh = --left == 0;
        if (fresh) {
            walk.next_rows();
            left = walk.run();
        }
        const uint64_t tile = b_desc + (stage * operand_bytes >> 4);
        uint64_t* const done_with = &empty_bar[stage];
        if (++stage == stages) stage = 0, parity ^= 1;
#pragma unroll
        for (uint32_t v = 0; v < 4; ++v) {  // halves of the rows by quarters of the columns
            const uint32_t u = 2 * v + first;
            emptied(v, i, bar, of);
            if (!wait(empty, bar, of, kWaitLimit)) return false;
            // the next waits are polled before this unit's products are issued, which hides their latency
            if (v == 3) full = mbar_test(&full_bar[stage], parity);
            emptied((v + 1) & 3, v == 3 ? i + 1 : i, bar, of);
            empty = mbar_test(bar, of);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elected) {
                const uint32_t at = first ? 4 + turn : v;
#pragma unroll
                for (int ks = 0; ks < KSTEPS; ++ks)
                    mma_f4(tmem + at * kUnitCols, tmem + kRowsAt + (v >> 1) * kRowsCols + ks * 8, tile + (u & 3) * ((kUnitCols * 16) >> 4) + ks * kStep,
                           tmem + kScalesAt, ks != 0);
                mma_commit(&tfull_bar[u]);
                if (v == 3) {
                    mma_commit(done_with);
                    if (fresh) mma_commit(done_bar);
                }
            }
            __syncwarp();
            if (++turn == 3) turn = 0;
        }
    }
    return true;
}

// QUADS: 16-byte words of a padded code row.  SECTIONS: there may be more hits than a list has room for
template <bool U16, int QUADS, bool SECTIONS>
__global__ void __launch_bounds__(kMmaThreads, 1) knn_mma_kernel(KnnMmaArgs a) {
    if (a.choice.skip()) return;
    extern __shared__ __align__(1024) unsigned char mma_smem[];
    __shared__ __align__(8) uint64_t full_bar[kMaxStages], empty_bar[kMaxStages];
    // of a step's units, not of the accumulators: who waits is then a phase behind at most
    __shared__ __align__(8) uint64_t tfull_bar[kUnitsStep], tempty_bar[kUnitsStep];
    __shared__ __align__(8) uint64_t rows_bar, done_bar;  // a row tile's rows are in tensor memory; its last products are through
    __shared__ __align__(8) uint64_t drain_bar;
    __shared__ __align__(16) uint4 hits_sm[SECTIONS ? 1 : kEpiWarps][8];
    __shared__ __align__(8) uint64_t met_bar, go_bar;
    __shared__ uint32_t listed, section, room;  // in the block's section, its number, and its room when the readers last met
    __shared__ uint32_t tmem_base_sm;
    __shared__ int abort_flag;
    const bool calm = a.calm.yes();
    if (calm && a.when == KnnMmaArgs::kNotIfCalm) return;
    const Phase phase = calm && a.when == KnnMmaArgs::kAllIfCalm ? Phase{a.phase.base, 1u, false, 0u, a.meet.columns() - a.phase.base} : a.phase;
    const int lane = threadIdx.x & 31, warp = __shfl_sync(kFull, int(threadIdx.x >> 5), 0);
    const uint32_t operand_bytes = uint32_t(a.chunks) * kMmaRows * 16;
    Walk walk(a.meet.row_tiles, phase.count);
    const uint32_t steps = walk.steps;

    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < kUnitsStep; ++i) {
            knn::mbar_init(&tfull_bar[i], 1);
            knn::mbar_init(&tempty_bar[i], 4);
        }
        for (int i = 0; i < kMaxStages; ++i) {
            knn::mbar_init(&full_bar[i], 1);
            knn::mbar_init(&empty_bar[i], kMmaWarps);
        }
        knn::mbar_init(&rows_bar, kEpiWarps);
        knn::mbar_init(&done_bar, kMmaWarps);
        knn::mbar_init(&drain_bar, kMmaWarps);
        knn::mbar_init(&met_bar, kEpiWarps);
        knn::mbar_init(&go_bar, 1);
        listed = 0, section = blockIdx.x;
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

    uint32_t loads = 0;  // tiles whose copies this warp has issued
    if (warp == kEpiWarps) {
        if (lane == 0) {
            uint32_t stage = 0, parity = 0;  // parity: of the stage's next filling
            bool ok = true;
            const unsigned char* op = reinterpret_cast<const unsigned char*>(a.operand);
            for (uint32_t i = 0; i < steps && !*aborted; ++i) {
                const uint32_t ct = a.meet.column(walk.rt, phase.column(walk.col));
                ok = wait_or_abort(&empty_bar[stage], parity ^ 1, a.handover_polls, aborted);  // handed back by the products
                if (!ok) break;
                knn::mbar_expect_tx(&full_bar[stage], operand_bytes);
                knn::bulk_g2s(mma_smem + stage * operand_bytes, op + size_t(ct) * operand_bytes, operand_bytes, &full_bar[stage]);
                ++loads;
                if (++stage == uint32_t(a.stages)) stage = 0, parity ^= 1;
                walk.next();
            }
            if (!ok) *aborted = 1;
        }
    } else if (warp > kEpiWarps) {
        const uint32_t elected = elect_one();
        auto issue = [&](auto ksteps) {
            return issue_products<decltype(ksteps)::value>(a, walk, steps, uint32_t(warp - kEpiWarps - 1), tmem, smem_u32(mma_smem), operand_bytes, elected, full_bar, empty_bar, tfull_bar,
                                                           tempty_bar, &rows_bar, &done_bar, aborted);
        };
        bool ok = false;
        switch (a.chunks) {
            case 2: ok = issue(std::integral_constant<int, 1>()); break;
            case 4: ok = issue(std::integral_constant<int, 2>()); break;
            case 6: ok = issue(std::integral_constant<int, 3>()); break;
            default: ok = issue(std::integral_constant<int, 4>()); break;
        }
        if (!ok) *aborted = 1;
        if (elected) mma_commit(&drain_bar);  // everything issued above has finished when this completes
    } else {
        const uint32_t quarter = warp & 3, cols = warp >> 2;  // of the lanes, of the columns
        const uint32_t addr = tmem + ((quarter * 32) << 16);
        // a part of a row tile's rows to tensor memory: the quarter of the first or second half, half of their chunks
        const uint32_t each = uint32_t(a.chunks) / 2, from = (cols >> 1) * each;
        auto put_rows = [&](uint32_t rt, bool again, uint32_t done_parity) {
            const uint4* src = a.operand + (size_t(rt) * a.chunks + from) * kMmaRows + (cols & 1) * 128 + quarter * 32 + lane;
            uint4 v[kRowsCols / 8];
#pragma unroll
            for (uint32_t c = 0; c < kRowsCols / 8; ++c)
                if (c < each) v[c] = __ldg(src + c * kMmaRows);
            if (again && !__all_sync(kFull, wait_or_abort(&done_bar, done_parity, kWaitLimit, aborted))) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (uint32_t c = 0; c < kRowsCols / 8; ++c)
                if (c < each && from + c < (kRowsCols - kScaleCols) / 4) tmem_store4(addr + kRowsAt + (cols & 1) * kRowsCols + (from + c) * 4, v[c]);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&rows_bar);
            return true;
        };
        if (cols < 2 && steps) tmem_store4(addr + kScalesAt + cols * kRowsCols, make_uint4(kScaleOne, kScaleOne, kScaleOne, kScaleOne));
        // the accumulators of the step's two units: two of the first warp's four, or those whose turn it is of the second's three
        uint32_t at0 = cols / 2, at1 = cols / 2 + 2, done_parity = 0;
        if (cols & 1) at0 += 4, at1 = at0 == 4 ? 6 : at0 - 1;
        // Hits are listed, and compared by a kernel behind the sweep.  One list: they wait in shared memory for a place in it, asked for
        // when more than four are there and used when the next come, or at the end: the place then has come (waiting for it took as
        // long as a step), and where hits are dense two steps' take one atomic on the list's length, which would be the bound there
        // (100k x 960, two bytes: two atomics a step 643 us, one 539; 100k x 64, K = 16, clusters of 100, the last phase: one 429,
        // with five to eight hits an atomic 272).
        uint4* const waiting = hits_sm[SECTIONS ? 0 : warp];
        uint32_t have = 0, asked = 0, to = 0;
        auto ask = [&]() {
            if (lane == 0) to = atomicAdd(a.hit_count, have);
            asked = have;
        };
        auto list_hits = [&]() {
            to = __shfl_sync(kFull, to, 0);
            if (uint32_t(lane) < asked) a.hits[to + lane] = waiting[lane];
            __syncwarp();
            have = asked = 0;
        };
        // Sections: a block fills one, with an atomic in shared memory for the place.  By the time that the section can be full the warps
        // meet, and the block goes on with it if it has room, with another one, or, when there are no others, after all its warps have
        // compared a part of what is in it.  (A warp that compares by itself what has no room holds up the others, which read the same
        // accumulators, and most warps have nothing to compare at that time.  Groups that overlap, sigma 0.45, K = 32, 64 neighbours:
        // 1M x 128 455 ms like that, 263 so; sigma 0.4, 16 neighbours, 2M 369 and 242.  Where hits are few the meetings are too: 1M,
        // sigma 0.3, 51.2 and 49.7.)  Up to 65,024 nodes every group has room in one list, which is quicker to go through (a check of
        // 14,000 x 300, two bytes, sigma 0.6: 676 us, 722 with sections).
        uint32_t next_look = SECTIONS ? kSection / kStepHits : ~0u, meetings = 0;
        auto meet = [&](auto then) {  // all of them, and what the first one does before any goes on
            __syncwarp();
            if (lane == 0) mbar_arrive(&met_bar);
            if (warp == 0) {
                if (!__all_sync(kFull, wait_or_abort(&met_bar, meetings & 1, kWaitLimit, aborted))) return false;
                if (lane == 0) {
                    then();
                    mbar_arrive(&go_bar);
                }
                __syncwarp();
            }
            return bool(__all_sync(kFull, wait_or_abort(&go_bar, meetings++ & 1, kWaitLimit, aborted)));
        };
        auto look = [&](uint32_t i) {
            const bool met = meet([&]() {
                room = kSection - listed;
                if (room >= kLeastRoom) return;
                const uint32_t other = a.blocks + atomicAdd(a.taken, 1u);
                room = 0;
                if (other >= kSections) return;
                a.section_hits[section] = listed;
                section = other, listed = 0, room = kSection;
            });
            if (!met) return false;
            if (room == 0) {
                const size_t first = size_t(section) * kSection;
#pragma unroll 1
                for (uint32_t e = listed - kDrain + warp; e < listed; e += kEpiWarps) compare_hit<U16, QUADS>(a, a.places[first + e], a.rows[first + e], lane);
                if (!meet([&]() { listed -= kDrain, room = kSection - listed; })) return false;
            }
            next_look = i + room / kStepHits;
            return true;
        };
        bool ok = true;
        for (uint32_t i = 0; i < steps && ok; walk.next_rows()) {
            const uint32_t rt = walk.rt, row0 = rt * kMmaRows + quarter * 32, run = min(walk.run(), steps - i);
            ok = put_rows(rt, i != 0, done_parity);
            if (i) done_parity ^= 1;
            // what a product reaches at the limit of the lane's row of either half, in the upper half
            const int least0 = gate_of(a.symbols, a.K, int(__ldg(a.place + row0 + lane).y)) << 16;
            const int least1 = gate_of(a.symbols, a.K, int(__ldg(a.place + row0 + 128 + lane).y)) << 16;
            // 32 steps' column tiles and what reaches the largest limit of their columns, a step a lane and asked for 32 ahead: a
            // pair is of use at the row's limit or at its column's, of which the largest of 32 stands for all at first
            uint32_t tile = 0, gates = 0, next_tile, next_gates;
            auto look_ahead = [&](uint32_t b) {
                next_tile = a.meet.column(rt, phase.column(walk.column(min(b + lane, run - 1))));
                next_gates = a.meet.both(rt, next_tile) ? __ldg(reinterpret_cast<const uint32_t*>(a.gate) + next_tile * 4 + cols) : 0x7fff7fffu;
            };
            look_ahead(0);
            for (uint32_t s = 0; s < run && ok; ++s, ++i) {
                if (SECTIONS && i == next_look && !look(i)) {
                    ok = false;
                    break;
                }
                if (s % 32 == 0) {
                    tile = next_tile, gates = next_gates;
                    if (s + 32 < run) look_ahead(s + 32);
                }
                const uint32_t pair = __shfl_sync(kFull, gates, s % 32);
                const int gate0 = int(pair << 16), gate1 = int(pair & 0xffff0000u);
                uint32_t rows[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    const uint32_t u = 4 * h + cols;
                    if (!__all_sync(kFull, knn::mbar_try_wait(&tfull_bar[u], i & 1)) &&
                        !__all_sync(kFull, wait_or_abort(&tfull_bar[u], i & 1, kWaitLimit, aborted))) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    uint32_t r[2][32];
                    const uint32_t from_col = addr + (h ? at1 : at0) * kUnitCols;
                    tmem_load32(r[0], from_col);
                    tmem_load32(r[1], from_col + 32);
                    tmem_wait(r[0], r[1]);
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&tempty_bar[u]);
                    // the largest product of every 32 columns
                    const int least = h ? least1 : least0;
                    const bool hit0 = largest(r[0]) >= min(least, gate0), hit1 = largest(r[1]) >= min(least, gate1);
                    rows[2 * h] = __ballot_sync(kFull, hit0);
                    rows[2 * h + 1] = __ballot_sync(kFull, hit1);
                }
                if (rows[0] | rows[1] | rows[2] | rows[3]) {
                    if (!SECTIONS && asked) list_hits();
                    const uint32_t some = (rows[0] != 0) | (rows[1] != 0) << 1 | (rows[2] != 0) << 2 | (rows[3] != 0) << 3;
                    const uint32_t ct = __shfl_sync(kFull, tile, s % 32);
                    if (SECTIONS) {
                        if (lane == 0) to = atomicAdd(&listed, uint32_t(__popc(some)));
                        to = __shfl_sync(kFull, to, 0);
                    }
                    if (some >> lane & 1u) {
                        const uint32_t mine = lane < 2 ? (lane ? rows[1] : rows[0]) : (lane == 2 ? rows[2] : rows[3]);
                        const uint32_t before = __popc(some & ((1u << lane) - 1u));
                        const uint32_t first_row = row0 + (lane >> 1) * 128, first_col = ct * kMmaRows + cols * kUnitCols + (lane & 1) * 32;
                        const uint32_t both = a.meet.both(rt, ct) ? 1u : 0u;
                        if (SECTIONS) {
                            const size_t at = size_t(section) * kSection + to + before;
                            a.places[at] = make_uint2(first_row | both, first_col);
                            a.rows[at] = mine;
                        } else {
                            waiting[have + before] = make_uint4(first_row, first_col, mine, both);
                        }
                    }
                    if (!SECTIONS) {
                        have += __popc(some);
                        __syncwarp();
                        if (have > 4) ask();
                    }
                }
                if (cols & 1) at1 = at0, at0 = at0 == 6 ? 4 : at0 + 1;
            }
        }
        if (!SECTIONS && have && !asked) ask();
        if (!SECTIONS && asked) list_hits();
        if (!ok) *aborted = 1;
    }
    __syncthreads();
    if (SECTIONS && threadIdx.x == 0) a.section_hits[section] = listed;
    // copies and products in flight after a lost wait end before the block's memory goes away
    if (*aborted && warp == kEpiWarps && lane == 0) {
        atomicExch(a.status, kStatusWaitTimeout);
        const uint32_t stages = uint32_t(a.stages);
        for (uint32_t l = loads > stages ? loads - stages : 0; l < loads; ++l) mbar_wait_bounded(&full_bar[l % stages], (l / stages) & 1, kWaitLimit);
    }
    if (warp == kEpiWarps + 1) {
        if (lane == 0) mbar_wait_bounded(&drain_bar, 0, kWaitLimit);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
    __syncthreads();
}

// ---- order of the nodes ----------------------------------------------------------------------------------------------
// A node's group is named by the smallest node among its likely neighbours, whose group is named the same way, followed to
// the end (nodes only get smaller; where it takes long, not to the end).  A cluster has a few such names; a node and its
// mate join theirs.
__device__ __forceinline__ uint32_t name_of(uint32_t* group, uint32_t node) {
    for (int i = 0; i < 64; ++i) {
        const uint32_t up = *reinterpret_cast<volatile uint32_t*>(group + node);
        if (up == node) break;
        node = up;
    }
    return node;
}
__global__ void group_join_kernel(uint32_t* __restrict__ group, const uint32_t* __restrict__ mate, uint32_t row_begin, uint32_t row_end,
                                  SweepChoice choice) {
    if (choice.skip()) return;
    const uint32_t row = row_begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= row_end) return;
    const uint32_t a = name_of(group, row), b = name_of(group, mate[row]);
    if (a != b) atomicMin(group + max(a, b), min(a, b));  // (one of several for the same name stays: the next round has the others)
}
__global__ void group_count_kernel(uint32_t* __restrict__ group, uint32_t row_begin, uint32_t row_end, uint32_t* __restrict__ count, SweepChoice choice) {
    if (choice.skip()) return;
    const uint32_t row = row_begin + blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t g = row < row_end ? name_of(group, row) : kInvalidNode;
    const uint32_t same = __match_any_sync(kFull, g);
    if (row >= row_end) return;
    group[row] = g;  // (a name on the same path: who reads it meanwhile gets there as well)
    if ((threadIdx.x & 31) == uint32_t(__ffs(same) - 1)) atomicAdd(count + g, uint32_t(__popc(same)));
}
// the places of the groups, in any order
__global__ void group_place_kernel(const uint32_t* __restrict__ count, uint32_t n, uint32_t* __restrict__ place, uint32_t* __restrict__ used,
                                   SweepChoice choice) {
    if (choice.skip()) return;
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const uint32_t c = g < n ? count[g] : 0u;
    uint32_t upto = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, upto, d);
        if (lane >= uint32_t(d)) upto += y;
    }
    uint32_t at = 0;
    if (lane == 31 && upto) at = atomicAdd(used, upto);
    at = __shfl_sync(kFull, at, 31) + upto - c;
    if (c) place[g] = at;
}
__global__ void group_scatter_kernel(const uint32_t* __restrict__ group, uint32_t row_begin, uint32_t row_end, uint32_t* __restrict__ place,
                                     uint32_t* __restrict__ node, SweepChoice choice) {
    if (choice.skip()) return;
    const uint32_t row = row_begin + blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const uint32_t g = row < row_end ? group[row] : kInvalidNode;
    const uint32_t same = __match_any_sync(kFull, g), first = __ffs(same) - 1;
    uint32_t at = 0;
    if (row < row_end && lane == first) at = atomicAdd(place + g, uint32_t(__popc(same)));
    at = __shfl_sync(kFull, at, first);
    if (row < row_end) node[at + __popc(same & ((1u << lane) - 1u))] = row;
}
// A block of 1,024 places: wanted rows, which come first (in their groups' order, or without one), a group's sorted by their limits; the other nodes behind the row
// tiles as they are; codes, limits and gates.
template <int QUADS>
__global__ void __launch_bounds__(kSortRows) layout_kernel(const uint4* __restrict__ codes, uint32_t n, uint32_t row_begin, uint32_t row_end,
                                                           const uint32_t* __restrict__ bound, const uint32_t* __restrict__ group, int K, int symbols, Meet meet,
                                                           const uint32_t* __restrict__ node, uint4* __restrict__ out, uint2* __restrict__ places,
                                                           int16_t* __restrict__ gate, SweepChoice choice) {
    if (choice.skip()) return;
    constexpr int kGates = kSortRows / 32, kGroups = 8, kLimits = 72;  // (groups from the eighth on are sorted together)
    __shared__ uint32_t cursor[kGroups * kLimits], begun[32];
    __shared__ int largest[kGates];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, chunk = blockIdx.x * kSortRows, place = chunk + tid;
    const uint32_t wanted = row_end - row_begin, behind = meet.row_tiles * kMmaRows;
    if (tid < kGroups * kLimits) cursor[tid] = 0;
    if (tid < kGates) largest[tid] = -1;
    uint32_t id = kInvalidNode, to = place, bin = 0;
    int lim = -1;
    bool begins = false;
    if (place < wanted) {
        id = node ? node[place] : row_begin + place;
        lim = int(min(bound[id], uint32_t(K)));
        begins = node && tid > 0 && group[id] != group[node[place - 1]];
    } else if (place >= behind && place - behind < n - wanted) {
        id = place - behind;
        if (id >= row_begin) id += wanted;
    }
    const uint32_t starts = __ballot_sync(kFull, begins);
    if (lane == 0) begun[warp] = __popc(starts);
    __syncthreads();
    if (lim >= 0) {
        uint32_t g = __popc(starts & (0xffffffffu >> (31 - lane)));
        for (uint32_t w = 0; w < warp; ++w) g += begun[w];
        bin = min(g, uint32_t(kGroups - 1)) * kLimits + uint32_t(lim);
        atomicAdd(&cursor[bin], 1u);
    }
    __syncthreads();
    if (warp == 0) {  // exclusive
        constexpr int kEach = kGroups * kLimits / 32;
        uint32_t x = 0;
        for (int i = 0; i < kEach; ++i) x += cursor[lane * kEach + i];
        const uint32_t own = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, x, o);
            if (lane >= uint32_t(o)) x += y;
        }
        x -= own;
        for (int i = 0; i < kEach; ++i) {
            const uint32_t c = cursor[lane * kEach + i];
            cursor[lane * kEach + i] = x;
            x += c;
        }
    }
    __syncthreads();
    if (lim >= 0) {
        const uint32_t rank = atomicAdd(&cursor[bin], 1u);
        to = chunk + rank;
        atomicMax(&largest[rank / 32], lim);
    }
    __syncthreads();
    if (to < meet.tiles * kMmaRows) {
        places[to] = make_uint2(id, uint32_t(lim));
#pragma unroll
        for (int w = 0; w < QUADS; ++w) out[size_t(to) * QUADS + w] = id != kInvalidNode ? __ldg(codes + size_t(id) * QUADS + w) : make_uint4(0u, 0u, 0u, 0u);
    }
    if (tid < kGates && chunk + tid * 32 < meet.row_tiles * kMmaRows) gate[chunk / 32 + tid] = int16_t(gate_of(symbols, K, largest[tid]));
}

// ---- buffers of more than kMmaCap entries, of one word each -----------------------------------------------------------
constexpr int kBins = 96;  // distances are 64 at most
struct Best {
    uint32_t T, last;  // the k-th distance; the largest node to take at it
};
// The k best of a buffer of more than k entries, or all up to the k-th distance where those are kMmaCap at most.  By the
// whole warp; bins: [kBins] of its own.
__device__ __forceinline__ Best best_of_long(const uint32_t* buf, uint32_t count, uint32_t k, uint32_t nodes, uint32_t* bins, int lane) {
    for (int i = lane; i < kBins; i += 32) bins[i] = 0;
    __syncwarp();
#pragma unroll 4
    for (uint32_t e = lane; e < count; e += 32) atomicAdd(bins + load_entry(buf, false, e).d, 1u);
    __syncwarp();
    const uint32_t c0 = bins[3 * lane], c1 = bins[3 * lane + 1], c2 = bins[3 * lane + 2];
    uint32_t upto = c0 + c1 + c2;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, upto, o);
        if (lane >= o) upto += y;
    }
    const int at = __ffs(__ballot_sync(kFull, upto >= k)) - 1;  // (count > k: there is one)
    uint32_t below = upto - c0 - c1 - c2, T = 3 * lane, same = c0;
    if (below + same < k) below += c0, same = c1, ++T;
    if (below + same < k) below += c1, same = c2, ++T;
    T = __shfl_sync(kFull, T, at), below = __shfl_sync(kFull, below, at), same = __shfl_sync(kFull, same, at);
    __syncwarp();
    if (below + same <= kMmaCap) return Best{T, kInvalidNode};
    uint32_t lo = 0, hi = nodes;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        uint32_t c = 0;
#pragma unroll 4
        for (uint32_t e = lane; e < count; e += 32) {
            const Entry x = load_entry(buf, false, e);
            c += x.d == T && x.node <= mid;
        }
        if (__reduce_add_sync(kFull, c) >= k - below) hi = mid;
        else lo = mid + 1;
    }
    return Best{T, lo};
}

// ---- between two phases: room in the buffers, limits of the k best so far ---------------------------------
// Where a buffer ran over the k-th distance of what it holds is a limit that few nodes are within: with a list the buffer
// starts anew and the row is listed for knn_again_kernel (without one nothing more is of use to the row for now).
// SHARE warps deal 32 rows among them: eight where the warps that took all 32 would be waited for (64 neighbours, sigma 0.3,
// 40,000 x 128: 1,057 us with one, 881 with eight), one in large graphs, whose warps are many and mostly have nothing to do.
// LONG: there are buffers of more than kMmaCap entries (the code for them costs those without it: 500,000 x 128 0.42 and 0.52 ms).
template <int SHARE, bool LONG>
__global__ void __launch_bounds__(kMmaRows) tighten_kernel(KnnMmaArgs a, bool only_lost, uint32_t* __restrict__ again /* places */,
                                                           uint32_t* __restrict__ again_count) {
    static_assert(SHARE == 1 || SHARE * 32 == kMmaRows, "a block has the rows of one gate, or a warp has");
    if (a.choice.skip() || (a.when == KnnMmaArgs::kNotIfCalm && a.calm.yes())) return;
    __shared__ uint32_t bins_sm[LONG ? kMmaRows / 32 : 1][kBins];
    __shared__ int largest;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t row0 = (blockIdx.x * (kMmaRows / 32) + warp) / SHARE * 32, own = row0 + lane;
    uint32_t count = a.counts[own];
    int limit = int(a.place[own].y);
    if constexpr (SHARE > 1) {
        if (threadIdx.x == 0) largest = -1;
        __syncthreads();  // (a row's own warp writes what the others have read)
    }
    const bool mine = SHARE == 1 || lane % SHARE == warp;
    const bool lost = count > a.cap, anew = lost && again;
    if (only_lost && !__any_sync(kFull, anew)) return;
    uint32_t todo = __ballot_sync(kFull, mine && (anew || (!lost && !only_lost && count >= a.k && limit >= 0)));
    const uint32_t anews = __ballot_sync(kFull, anew);
    while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        uint32_t c = min(__shfl_sync(kFull, count, src), a.cap);
        uint32_t* buf = buffer_of(a, row0 + src);
        uint32_t T;
        auto kth = [&](auto slots) {
            uint32_t dist[decltype(slots)::value];
#pragma unroll
            for (int s = 0; s < decltype(slots)::value; ++s) dist[s] = uint32_t(s * 32 + lane) < c ? load_entry(buf, a.wide, s * 32 + lane).d : kFull;
            return kth_distance(dist, a.k, a.K);
        };
        if (LONG && c > kMmaCap) {
            const Best best = best_of_long(buf, c, a.k, a.meet.tiles * kMmaRows, bins_sm[warp], lane);
            T = best.T;
            if (!(anews >> src & 1u)) c = keep_entries(buf, false, c, T, best.last, lane);
        } else if (!(anews >> src & 1u) && c > kMmaFull) T = compact_row(buf, a.wide, c, a.k, a.K, lane);
        else if (c > kMmaFull) T = kth(std::integral_constant<int, kMmaSlots>());
        else if (c > kMmaKeep) T = kth(std::integral_constant<int, kMmaFull / 32>());
        else T = kth(std::integral_constant<int, kMmaKeep / 32>());
        if (anews >> src & 1u) c = 0;
        if (lane == src) count = c, limit = limit < 0 || limit > int(T) ? int(T) : limit;
    }
    if (mine) {
        if (anew) again[atomicAdd(again_count, 1u)] = own;
        if (lost && !again) limit = -1;
        a.counts[own] = count;
        a.place[own].y = uint32_t(limit);
    }
    int most = __reduce_max_sync(kFull, mine ? limit : -1);
    if constexpr (SHARE > 1) {
        if (lane == 0) atomicMax(&largest, most);
        __syncthreads();
        most = largest;
    }
    if (SHARE == 1 ? lane == 0 : threadIdx.x == 0) a.gate[row0 / 32] = int16_t(gate_of(a.symbols, a.K, most));
}

// The listed rows against the nodes of all tiles, or of the row tiles less than `near` tiles away, at their new limits; grid
// y deals the rows, grid x the nodes.
template <bool U16, int QUADS>
__global__ void __launch_bounds__(256) knn_again_kernel(KnnMmaArgs a, const uint32_t* __restrict__ again, const uint32_t* __restrict__ again_count,
                                                        uint32_t near) {
    if (a.choice.skip()) return;
    const uint32_t many = *again_count, places = (near ? 2 * near - 1 : a.meet.tiles) * kMmaRows;
    for (uint32_t b = blockIdx.y; b < many; b += gridDim.y) {
        const uint32_t row = again[b], tile = row / kMmaRows;
        const uint32_t from = near ? (tile >= near - 1 ? tile - (near - 1) : tile + a.meet.row_tiles - (near - 1)) * kMmaRows : 0;
        const int limit = int(a.place[row].y);
        uint4 own[QUADS];
#pragma unroll
        for (int w = 0; w < QUADS; ++w) own[w] = __ldg(a.codes + size_t(row) * QUADS + w);
#pragma unroll 4
        for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < places; i += gridDim.x * 256) {
            uint32_t j = from + i;
            if (near && j >= a.meet.row_tiles * kMmaRows) j -= a.meet.row_tiles * kMmaRows;
            uint4 v[QUADS];
#pragma unroll
            for (int w = 0; w < QUADS; ++w) v[w] = __ldg(a.codes + size_t(j) * QUADS + w);
            const int d = int(code_distance<U16, QUADS>(own, v));
            if (d > limit || j == row) continue;
            const uint32_t node = a.place[j].x;
            if (node == kInvalidNode) continue;
            const uint32_t at = atomicAdd(a.counts + row, 1u);
            if (at < a.cap) store_entry(buffer_of(a, row), a.wide, at, uint32_t(d), node);
        }
    }
}

// ---- results: the k best of a row's buffer by (distance, id) -----------------------------------------------------------
// A warp a row.  The entries up to the k-th distance, k and a few ties, are sorted in registers as the words they are; where
// they are wide or many, a row's rank is the number of entries before it.
constexpr int kFinishWarps = 4;
constexpr int kFinishSort = 128;
__global__ void __launch_bounds__(kFinishWarps * 32) knn_finish_kernel(KnnMmaArgs a, uint32_t rows, uint32_t* __restrict__ nbrs,
                                                                       uint16_t* __restrict__ dists, uint32_t out_row0,
                                                                       uint32_t* __restrict__ redo /* rows */, uint32_t* __restrict__ redo_count) {
    if (a.choice.skip()) return;
    __shared__ uint64_t keys_sm[kFinishWarps][kMmaCap];
    __shared__ uint32_t bins_sm[kFinishWarps][kBins];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t place = blockIdx.x * kFinishWarps + warp;
    if (place >= rows) return;
    const uint32_t row = a.place[place].x, count = a.counts[place];
    if (row == kInvalidNode) return;
    if (count > a.cap) {
        if (lane == 0) redo[atomicAdd(redo_count, 1u)] = row;
        return;
    }
    const uint32_t* buf = buffer_of(a, place);
    uint32_t* out_n = nbrs + size_t(row - out_row0) * a.k;
    uint16_t* out_d = dists ? dists + size_t(row - out_row0) * a.k : nullptr;
    uint64_t* keys = keys_sm[warp];
    uint32_t* words = reinterpret_cast<uint32_t*>(keys);
    const uint32_t below = (1u << lane) - 1u;
    uint32_t m = 0;
    if (count > kMmaCap) {
        const Best best = best_of_long(buf, count, a.k, a.meet.tiles * kMmaRows, bins_sm[warp], lane);
#pragma unroll 4
        for (uint32_t e0 = 0; e0 < count; e0 += 32) {
            const Entry x = e0 + lane < count ? load_entry(buf, false, e0 + lane) : Entry{kFull, 0u};
            const bool take = x.d < best.T || (x.d == best.T && x.node <= best.last);
            const uint32_t b = __ballot_sync(kFull, take);
            if (take) words[m + __popc(b & below)] = x.d << 25 | x.node;
            m += __popc(b);
        }
    } else {
        Entry x[kMmaSlots];
        uint32_t dist[kMmaSlots];
#pragma unroll
        for (int s = 0; s < kMmaSlots; ++s) {
            x[s] = Entry{kFull, 0u};
            if (s * 32u < count && uint32_t(s * 32 + lane) < count) x[s] = load_entry(buf, a.wide, s * 32 + lane);
            dist[s] = x[s].d;
        }
        uint32_t T = uint32_t(a.K);
        if (count > a.k) {
            if (count <= kMmaKeep) T = kth_distance(reinterpret_cast<const uint32_t (&)[kMmaKeep / 32]>(dist), a.k, a.K);
            else T = kth_distance(dist, a.k, a.K);
        }
#pragma unroll
        for (int s = 0; s < kMmaSlots; ++s) {
            if (s * 32u >= count) break;
            const bool take = x[s].d <= T;
            const uint32_t b = __ballot_sync(kFull, take), at = m + __popc(b & below);
            if (take && a.wide) keys[at] = (uint64_t(x[s].d) << 32) | x[s].node;
            else if (take) words[at] = x[s].d << 25 | x[s].node;
            m += __popc(b);
        }
    }
    __syncwarp();
    const uint32_t kept = min(m, a.k);
    if (!a.wide && m <= uint32_t(kFinishSort)) {
        uint32_t v[kFinishSort / 32];  // element s * 32 + lane
#pragma unroll
        for (int s = 0; s < kFinishSort / 32; ++s) v[s] = uint32_t(s * 32 + lane) < m ? words[s * 32 + lane] : kFull;
#pragma unroll
        for (int size = 2; size <= kFinishSort; size *= 2) {
#pragma unroll
            for (int d = size / 2; d >= 1; d /= 2) {
                if (d >= 32) {
#pragma unroll
                    for (int s = 0; s < kFinishSort / 32; ++s) {
                        if (s & (d / 32)) continue;
                        const bool up = ((s * 32) & size) == 0;  // (the whole is ascending: no bit at its size)
                        const uint32_t lo = min(v[s], v[s | (d / 32)]), hi = max(v[s], v[s | (d / 32)]);
                        v[s] = up ? lo : hi, v[s | (d / 32)] = up ? hi : lo;
                    }
                } else {
#pragma unroll
                    for (int s = 0; s < kFinishSort / 32; ++s) {
                        const uint32_t y = __shfl_xor_sync(kFull, v[s], d);
                        const bool low = ((lane & d) == 0) == (((s * 32 + lane) & size) == 0);
                        v[s] = low ? min(v[s], y) : max(v[s], y);
                    }
                }
            }
        }
#pragma unroll
        for (int s = 0; s < kFinishSort / 32; ++s) {
            const uint32_t rank = s * 32 + lane;
            if (rank >= kept) continue;
            out_n[rank] = v[s] & (kPackedNodes - 1u);
            if (out_d) out_d[rank] = uint16_t(v[s] >> 25);
        }
    } else {
        for (uint32_t e = lane; e < m; e += 32) {
            auto key = [&](uint32_t i) { return a.wide ? keys[i] : (uint64_t(words[i] >> 25) << 32) | (words[i] & (kPackedNodes - 1u)); };
            const uint64_t own = key(e);
            uint32_t rank = 0;
            for (uint32_t i = 0; i < m; ++i) rank += key(i) < own;
            if (rank >= kept) continue;
            out_n[rank] = uint32_t(own);
            if (out_d) out_d[rank] = uint16_t(own >> 32);
        }
    }
    for (uint32_t o = kept + lane; o < a.k; o += 32) {
        out_n[o] = kInvalidNode;
        if (out_d) out_d[o] = 0xFFFF;
    }
}

// ---- rows whose buffer ran over: compared with every node ---------------------------------------------------------------
// A block a row, twice over the nodes: the distances up to the row's bound are counted, then the nodes below the k-th are
// collected, and the smallest ids at it, which every warp finds first in its own range of the nodes.
constexpr int kRedoWarps = 32;
template <bool U16, int QUADS>
__global__ void __launch_bounds__(kRedoWarps * 32) knn_redo_kernel(const uint4* __restrict__ codes, uint32_t n, uint32_t k, int K,
                                                                   const uint32_t* __restrict__ bound, const uint32_t* __restrict__ redo,
                                                                   const uint32_t* __restrict__ redo_count,
                                                                   uint32_t* __restrict__ nbrs, uint16_t* __restrict__ dists, uint32_t out_row0,
                                                                   SweepChoice choice) {
    if (choice.skip()) return;
    __shared__ uint32_t hist[96], ties[kRedoWarps][128], tie_count[kRedoWarps], below_sm, T_sm, found;
    __shared__ uint64_t keys[128];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, many = *redo_count;
    const uint32_t from = uint32_t(uint64_t(n) * warp / kRedoWarps), to = uint32_t(uint64_t(n) * (warp + 1) / kRedoWarps);
    for (uint32_t b = blockIdx.x; b < many; b += gridDim.x) {
        const uint32_t row = redo[b], most = min(bound[row], uint32_t(K));
        uint4 own[QUADS];
#pragma unroll
        for (int w = 0; w < QUADS; ++w) own[w] = __ldg(codes + size_t(row) * QUADS + w);
        auto distance = [&](uint32_t j) {
            uint4 v[QUADS];
#pragma unroll
            for (int w = 0; w < QUADS; ++w) v[w] = __ldg(codes + size_t(j) * QUADS + w);
            return code_distance<U16, QUADS>(own, v);
        };
        if (tid < 96) hist[tid] = 0;
        if (tid == 0) found = 0;
        __syncthreads();
#pragma unroll 4
        for (uint32_t j0 = from; j0 < to; j0 += 32) {
            const uint32_t j = j0 + lane, d = j < to && j != row ? distance(j) : kFull;
            // one addition for the lanes at the lowest distance of the step, one each for the others
            const uint32_t low = __reduce_min_sync(kFull, d), same = __ballot_sync(kFull, d == low);
            if (low > most) continue;
            if (d == low ? lane == uint32_t(__ffs(same) - 1) : d <= most) atomicAdd(hist + d, d == low ? uint32_t(__popc(same)) : 1u);
        }
        __syncthreads();
        if (tid == 0) {
            uint32_t T = 0, below = 0;
            while (T < most && below + hist[T] < k) below += hist[T++];
            T_sm = T, below_sm = below;
        }
        __syncthreads();
        const uint32_t T = T_sm, below = below_sm, need = k - below;  // need >= 1 of those at T (or all there are)
        uint32_t have = 0;
#pragma unroll 4
        for (uint32_t j0 = from; j0 < to; j0 += 32) {
            const uint32_t j = j0 + lane, d = j < to && j != row ? distance(j) : kFull;
            if (d < T) keys[atomicAdd(&found, 1u)] = (uint64_t(d) << 32) | j;
            const uint32_t m = __ballot_sync(kFull, d == T);
            const uint32_t at = have + __popc(m & ((1u << lane) - 1u));
            if (d == T && at < need) ties[warp][at] = j;
            have = min(need, have + uint32_t(__popc(m)));
        }
        if (lane == 0) tie_count[warp] = have;
        __syncthreads();
        uint32_t skip = 0;  // ties of the warps before
        for (uint32_t w = 0; w < warp; ++w) skip += tie_count[w];
        for (uint32_t i = lane; i < have && skip + i < need; i += 32) keys[below + skip + i] = (uint64_t(T) << 32) | ties[warp][i];
        uint32_t total = 0;
        for (uint32_t w = 0; w < kRedoWarps; ++w) total += tie_count[w];
        total = below + min(need, total);
        __syncthreads();
        uint32_t* out_n = nbrs + size_t(row - out_row0) * k;
        uint16_t* out_d = dists ? dists + size_t(row - out_row0) * k : nullptr;
        if (tid < k) {
            uint32_t rank = tid, id = kInvalidNode, d = 0xFFFF;
            if (tid < total) {
                const uint64_t key = keys[tid];
                rank = 0, id = uint32_t(key), d = uint32_t(key >> 32);
                for (uint32_t i = 0; i < total; ++i) rank += keys[i] < key;
            }
            out_n[rank] = id;
            if (out_d) out_d[rank] = uint16_t(d);
        }
        __syncthreads();
    }
}

template <typename CompT, int QUADS>
int launch_mma_t(cphnsw_b200_index* h, const void* d_codes, const uint32_t* padded, uint64_t n, uint32_t k, uint64_t row_begin,
                 uint64_t row_end, uint32_t* d_nbrs, uint16_t* d_dist, double most_turns, SweepChoice* other, cudaStream_t st) {
    constexpr bool U16 = sizeof(CompT) == 2;
    const CompT* codes = static_cast<const CompT*>(d_codes);
    const uint4* rows = reinterpret_cast<const uint4*>(padded);
    const HashShape shape = hash_shape(int(h->K));
    const uint32_t operand_bytes = uint32_t(shape.chunks) * kMmaRows * 16;
    const uint32_t sms = uint32_t(h->sm_count);
    const uint64_t wanted = row_end - row_begin;
    // (places are words of 32 bits, rounded up by tiles; at 144 bytes a node and more no GPU this runs on has room for as many)
    if (n > uint64_t(1) << 31) return kNoRoom;

    // Workspace.  The buffers take 1.5 KB a wanted row, 3 KB with entries of two words: where they do not fit, the rows go in
    // blocks.
    auto up = [](size_t b) { return (b + 255) & ~size_t(255); };
    const uint64_t most_tiles = (n + kMmaRows - 1) / kMmaRows + 1;  // row tiles and the others are rounded up apart
    const size_t op_b = up(size_t(most_tiles) * operand_bytes), codes_b = up(size_t(most_tiles) * kMmaRows * QUADS * 16);
    const size_t places_b = up(size_t(most_tiles) * kMmaRows * 8), gates_b = up(size_t(most_tiles) * 16), n_b = up(size_t(n) * 4);
    const size_t hist_b = up(size_t(kBoundOrders) * kKeys * 4), order_b = up(size_t(kBoundOrders) * n * 4);
    const size_t before_b = hist_b + 2 * order_b;  // of use until the sweep begins, in the buffers' place
    uint64_t block = wanted;
    const bool wide = n > kPackedNodes - 1;  // (the last packed node stands for none)
    const uint64_t most_hits = most_tiles * (most_tiles + 1) * kStepHits;  // (a launch has no more steps)
    const bool sections = most_hits > kHitRoom;
    const size_t hits_b = up(sections ? size_t(kSections) * kSection * 8 : size_t(most_hits) * 16);
    const size_t rows_b = sections ? up(size_t(kSections) * kSection * 4) : 0, section_hits_b = up(kSections * 4);
    size_t entries_b, counts_b, list_b;
    // In one phase a row's limit stays what the places beside it say, the k-th of 512 distances: on data without clusters a
    // share of k / 512 of the nodes is within it, which twice as long a buffer holds with the ties.  (With 384 entries nearly
    // every row ran over and was compared with all nodes up to three times more; K = 32, unit sphere, 5,000 nodes: 716 us so,
    // 319 now; K = 64, 8,191 nodes: 2,048 and 715; mixture of sigma 0.6, 14,000 x 960, two bytes: 2,598 and 1,378.  Clustered
    // data do not touch what they do not fill.  Components of two bytes have so many values that without
    // clusters nearly all distances are K: buffers twice as long hold enough of those that are not; 300-d, unit sphere, 8,191
    // nodes 2,696 us and 1,388, 7,000 2,058 and 1,086.)
    const Meet whole{uint32_t((wanted + kMmaRows - 1) / kMmaRows + (n - wanted + kMmaRows - 1) / kMmaRows), uint32_t((wanted + kMmaRows - 1) / kMmaRows)};
    uint64_t cap = kMmaCap;
    const bool small = whole.columns() <= kOnePhase && whole.row_tiles / 2 + 1 < kNearFrom;
    if (small) {
        const uint64_t longest = kLongBuffers / (uint64_t(whole.row_tiles) * kMmaRows * 4), of_use = n * k / (U16 ? 128 : 256);
        cap = (of_use < longest ? of_use : longest) / 32 * 32;
        if (cap < kMmaCap) cap = kMmaCap;
    }
    while (true) {
        const size_t slots = size_t((block + kMmaRows - 1) / kMmaRows) * kMmaRows;
        entries_b = up(slots * cap * (wide ? 8 : 4)), counts_b = up(slots * 4), list_b = up(slots * 4);
        const size_t buffers_b = entries_b > before_b ? entries_b : before_b;
        const int rc = reserve_workspace(h, h->s_sliced, op_b + codes_b + places_b + gates_b + 6 * n_b + buffers_b + counts_b + 2 * list_b + hits_b + rows_b + section_hits_b + 512);
        if (rc == 0) break;
        if (rc == kNoRoom && cap > kMmaCap) {
            cap = kMmaCap;
            continue;
        }
        if (rc != kNoRoom || entries_b <= before_b || block <= uint64_t(sms) * kMmaRows) return rc;
        block = (block + 1) / 2;
    }
    KnnMmaArgs a;
    unsigned char* p = h->s_sliced.as<unsigned char>();
    auto take = [&](size_t b) {
        unsigned char* r = p;
        p += b;
        return r;
    };
    uint4* operand = reinterpret_cast<uint4*>(take(op_b));
    uint4* placed = reinterpret_cast<uint4*>(take(codes_b));
    uint2* places = reinterpret_cast<uint2*>(take(places_b));
    int16_t* gate = reinterpret_cast<int16_t*>(take(gates_b));
    uint32_t* bound = reinterpret_cast<uint32_t*>(take(n_b));
    uint32_t* group = reinterpret_cast<uint32_t*>(take(n_b));
    uint32_t* mate = reinterpret_cast<uint32_t*>(take(n_b));
    uint32_t* far = mate;  // rows whose bound says little (the mates have joined their groups by then)
    uint32_t* grouped = reinterpret_cast<uint32_t*>(take(n_b));
    uint32_t* group_place = reinterpret_cast<uint32_t*>(take(n_b));
    uint32_t* again = reinterpret_cast<uint32_t*>(take(list_b));
    uint32_t* redo = reinterpret_cast<uint32_t*>(take(list_b));
    a.hits = reinterpret_cast<uint4*>(p);
    a.places = reinterpret_cast<uint2*>(take(hits_b));
    a.rows = reinterpret_cast<uint32_t*>(take(rows_b));
    a.section_hits = reinterpret_cast<uint32_t*>(take(section_hits_b));
    // cleared for every block of rows, in one go (as clears of their own: a graph of 4,096 nodes 177 us, 167 so)
    struct Counters {
        uint32_t used, hits, far, again, redo;  // hits: or sections taken
    };
    static_assert(sizeof(Counters) <= 256 && sizeof(LoadCounts) <= 256, "counters take 256 bytes");
    unsigned char* cleared = p;
    Counters* counters = reinterpret_cast<Counters*>(take(256));
    uint32_t* group_count = reinterpret_cast<uint32_t*>(take(n_b));
    uint32_t* counts = reinterpret_cast<uint32_t*>(take(counts_b));
    LoadCounts* load = reinterpret_cast<LoadCounts*>(take(256));
    uint32_t* entries = reinterpret_cast<uint32_t*>(p);
    uint32_t* hist = reinterpret_cast<uint32_t*>(take(hist_b));
    uint32_t* order = reinterpret_cast<uint32_t*>(take(order_b));
    uint32_t* place = reinterpret_cast<uint32_t*>(take(order_b));

    // data that are not calm, in small graphs: bounds and near columns as in larger ones
    const bool two = small && other && whole.row_tiles / 2 + 1 >= 2 * kNearColumns;
    a.operand = operand;
    a.codes = placed;
    a.place = places;
    a.gate = gate;
    a.wide = wide;
    a.cap = uint32_t(cap);
    a.K = int(h->K);
    a.symbols = shape.symbols;
    a.chunks = shape.chunks;
    a.stages = int(kMmaSmem / operand_bytes);
    if (a.stages > kMaxStages) a.stages = kMaxStages;
    // (never two blocks on an SM, of which the second would wait for the first one's tensor memory)
    const size_t ring = size_t(a.stages) * operand_bytes, sweep_smem = ring > (size_t(120) << 10) ? ring : size_t(120) << 10;
    a.k = k;
    a.entries = entries;
    a.counts = counts;
    a.hit_count = a.taken = &counters->hits;
    a.status = h->d_status.as<uint32_t>();
    a.first_wait_polls = h->first_wait_polls;
    a.handover_polls = h->handover_polls;

    LoadArgs sample;
    sample.groups = uint32_t((wanted + 31) / 32 < kLoadGroups ? (wanted + 31) / 32 : kLoadGroups);
    sample.apart = wanted / sample.groups < 32 ? 32 : wanted / sample.groups;
    const uint64_t node_tiles = (n + kMmaRows - 1) / kMmaRows;
    if (other) {
        a.choice.load = &load->turns;
        a.choice.most = (unsigned long long)(most_turns * sample.groups * kLoadTiles);
        *other = a.choice;
        other->above = true;
        a.calm.counts = load;
        a.calm.most_turns = (unsigned long long)((two ? kSmallCalm / (double(n) * n) * (QUADS > 2 ? 0.56 : 1.0) : kCalmTurns) * sample.groups * kLoadTiles);
        a.calm.most = two ? kFull : uint32_t(kCalmEntries * 32 * kLoadTiles * sample.groups / double(node_tiles));
    }
    CPB_CUDA(cudaMemsetAsync(load, 0, 256 + hist_b, st));
    const dim3 by_row(unsigned((n + 255) / 256), kBoundOrders);
    key_count_kernel<CompT><<<by_row, 256, 0, st>>>(codes, n, int(h->K), hist);
    key_scan_kernel<<<kBoundOrders, 1024, 0, st>>>(hist);
    key_scatter_kernel<CompT><<<by_row, 256, 0, st>>>(codes, n, int(h->K), hist, order, place);
    auto bounds = [&](uint64_t count, uint64_t apart, auto orders, auto window, const uint32_t* listed, const SweepChoice& choice, const Calm& calm = Calm()) {
        auto go = [&](auto kernel) {
            kernel<<<unsigned((count + kBoundWarps - 1) / kBoundWarps), kBoundWarps * 32, 0, st>>>(rows, a.K, n, order, place, k, uint32_t(row_begin),
                                                                                                  uint32_t(row_end), bound, group, mate, apart, listed, &counters->far, choice, calm);
        };
        constexpr int O = decltype(orders)::value, W = decltype(window)::value;
        if (QUADS > 1 && reinterpret_cast<uintptr_t>(padded) % 32 == 0) go(bound_kernel<U16, QUADS, (QUADS > 1), O, W>);
        else go(bound_kernel<U16, QUADS, false, O, W>);
        h->launches++;
    };
    using All = std::integral_constant<int, kBoundOrders>;
    using Full = std::integral_constant<int, kBoundWindow>;
    if (other) {
        bounds(uint64_t(sample.groups) * 32, sample.apart, All(), Full(), nullptr, SweepChoice());
        load_kernel<U16, QUADS><<<dim3(sample.groups, kLoadTiles), kMmaRows, 0, st>>>(rows, n, uint32_t(shape.symbols), uint32_t(node_tiles),
                                                                                     uint32_t(row_begin), uint32_t(row_end), bound, sample,
                                                                                     load);
        h->launches++;
    }
    const bool ordered = n >= kOrderNodes;
    if (ordered) bounds(n, 0, std::integral_constant<int, kNameOrders>(), std::integral_constant<int, kNameWindow>(), nullptr, a.choice);
    else bounds(n, 0, All(), std::integral_constant<int, kBoundWindow / 2>(), nullptr, a.choice);
    const unsigned row_blocks = unsigned((wanted + 255) / 256);
    for (int i = 0; i < (n > kOnePhase * 2 * kMmaRows ? 3 : 2) && ordered; ++i) group_join_kernel<<<row_blocks, 256, 0, st>>>(group, mate, uint32_t(row_begin), uint32_t(row_end), a.choice);
    h->launches += ordered ? 6 : 3;
    CPB_CUDA(cudaGetLastError());
    CPB_CUDA(allow_max_dynamic_smem(beside_kernel<U16, QUADS>));
    if (sections) CPB_CUDA(allow_max_dynamic_smem(knn_mma_kernel<U16, QUADS, true>));
    else CPB_CUDA(allow_max_dynamic_smem(knn_mma_kernel<U16, QUADS, false>));
    const uint32_t most_blocks = sms < kSections ? sms : kSections;
    for (uint64_t begin = row_begin; begin < row_end; begin += block) {
        const uint32_t rb = uint32_t(begin), re = uint32_t(row_end - begin < block ? row_end : begin + block), m = re - rb;
        a.meet.row_tiles = (m + kMmaRows - 1) / kMmaRows;
        a.meet.tiles = a.meet.row_tiles + uint32_t((n - m + kMmaRows - 1) / kMmaRows);
        // (a block that gives up leaves rows without entries: they are then empty, not whatever the workspace held)
        CPB_CUDA(cudaMemsetAsync(cleared, 0, 256 + n_b + size_t(a.meet.row_tiles) * kMmaRows * 4, st));
        if (ordered) {
            group_count_kernel<<<(m + 255) / 256, 256, 0, st>>>(group, rb, re, group_count, a.choice);
            group_place_kernel<<<unsigned((n + 255) / 256), 256, 0, st>>>(group_count, uint32_t(n), group_place, &counters->used, a.choice);
            group_scatter_kernel<<<(m + 255) / 256, 256, 0, st>>>(group, rb, re, group_place, grouped, a.choice);
            beside_kernel<U16, QUADS><<<(m + kBesideRows - 1) / kBesideRows, kBesideWarps * 32,
                                        kBesidePlaces * QUADS * 16 + (a.K + 1) * kBesideWarps * 64, st>>>(rows, grouped, m, a.K, k, bound, far, &counters->far, a.choice);
            // (the orders are still there for the first block of rows only)
            if (rb == row_begin && n > kOnePhase * 2 * kMmaRows) bounds(uint64_t(sms) * 64, 0, All(), Full(), far, a.choice);
            else if (rb == row_begin && two && whole.columns() > kOnePhaseBounds) bounds(uint64_t(sms) * 64, 0, All(), Full(), far, a.choice, a.calm);
            h->launches += 4;
        }
        layout_kernel<QUADS><<<(a.meet.tiles * kMmaRows + kSortRows - 1) / kSortRows, kSortRows, 0, st>>>(
            rows, uint32_t(n), rb, re, bound, group, a.K, a.symbols, a.meet, ordered ? grouped : nullptr, placed, places, gate, a.choice);
        const uint64_t cells = uint64_t(a.meet.tiles) * shape.chunks * kMmaRows;
        expand_codes_kernel<CompT><<<unsigned((cells + 255) / 256), 256, 0, st>>>(reinterpret_cast<const CompT*>(placed), QUADS * 16 / int(sizeof(CompT)),
                                                                                 places, int(h->K), shape.symbols, shape.chunks, operand,
                                                                                 a.meet.tiles, a.choice);
        h->launches += 2;
        const uint32_t columns = a.meet.columns();
        // A launch takes 4M steps: on clustered data, where nearly all of them have no hit, those there are have room in the sections.
        const uint32_t range = uint32_t(kLaunchSteps / a.meet.row_tiles) + 1;
        bool first = true;
        auto sweep = [&](uint32_t count) {
            const uint64_t steps = uint64_t(a.meet.row_tiles) * count;
            if (!first) CPB_CUDA(cudaMemsetAsync(a.hit_count, 0, 4, st));
            first = false;
            a.blocks = uint32_t(steps < most_blocks ? steps : most_blocks);
            if (sections) {
                knn_mma_kernel<U16, QUADS, true><<<a.blocks, kMmaThreads, sweep_smem, st>>>(a);
                knn_check_sections_kernel<U16, QUADS><<<sms * kCheckBlocks, kCheckWarps * 32, 0, st>>>(a);
            } else {
                knn_mma_kernel<U16, QUADS, false><<<a.blocks, kMmaThreads, sweep_smem, st>>>(a);
                knn_check_kernel<U16, QUADS><<<sms * kCheckBlocks, kCheckWarps * 32, 0, st>>>(a);
            }
            h->launches += 2;
            return 0;
        };
        auto tighten = [&](bool only_lost, uint32_t* list) {
            const unsigned shared = a.meet.row_tiles * 8;
            if (cap > kMmaCap) tighten_kernel<8, true><<<shared, kMmaRows, 0, st>>>(a, only_lost, list, &counters->again);
            else if (a.meet.row_tiles < 8 * sms) tighten_kernel<8, false><<<shared, kMmaRows, 0, st>>>(a, only_lost, list, &counters->again);
            else tighten_kernel<1, false><<<a.meet.row_tiles, kMmaRows, 0, st>>>(a, only_lost, list, &counters->again);
            h->launches++;
        };
        // near columns, among which a group's rows are
        uint32_t near = 0;
        if (a.meet.row_tiles / 2 + 1 >= kNearFrom) {
            near = kNearColumns;
            a.when = KnnMmaArgs::kAlways;
            a.phase = Phase{0u, 1u, false, 0u, near};
            CPB_TRY(sweep(near));
            tighten(false, again);
            knn_again_kernel<U16, QUADS><<<dim3(2, 4 * sms), 256, 0, st>>>(a, again, &counters->again, near);
            CPB_CUDA(cudaMemsetAsync(&counters->again, 0, 4, st));
            h->launches++;
        }
        if (two) {  // the same where data are not calm; the others take all columns at once
            near = kNearColumns;
            a.when = KnnMmaArgs::kAllIfCalm;
            a.phase = Phase{0u, 1u, false, 0u, near};
            CPB_TRY(sweep(columns));
            a.when = KnnMmaArgs::kNotIfCalm;
            tighten(false, again);
            knn_again_kernel<U16, QUADS><<<dim3(2, 4 * sms), 256, 0, st>>>(a, again, &counters->again, near);
            CPB_CUDA(cudaMemsetAsync(&counters->again, 0, 4, st));
            h->launches++;
        }
        uint32_t stride = 1;
        while (columns > kOnePhase && columns - near > kFirstColumns * stride) stride *= 2;
        const bool one = a.calm.counts && columns - near <= range;  // (does on calm data)
        for (bool whole = true; stride; stride /= 2, whole = false) {
            a.phase = Phase{near, stride, !whole, 0u, 0u};
            const uint32_t all = a.phase.columns(columns);
            for (uint32_t from = 0; from < all; from += range) {
                a.when = one ? (whole && from == 0 && !two ? KnnMmaArgs::kAllIfCalm : KnnMmaArgs::kNotIfCalm) : KnnMmaArgs::kAlways;
                a.phase.from = from, a.phase.count = all - from < range ? all - from : range;
                CPB_TRY(sweep(a.when == KnnMmaArgs::kAllIfCalm ? columns - near : a.phase.count));
            }
            if (stride > 1) {
                if (one) a.when = KnnMmaArgs::kNotIfCalm;
                tighten(false, nullptr);
            }
        }
        a.when = KnnMmaArgs::kAlways;
        tighten(true, again);
        knn_again_kernel<U16, QUADS><<<dim3(16, sms), 256, 0, st>>>(a, again, &counters->again, 0u);
        const uint32_t slots = a.meet.row_tiles * kMmaRows;
        knn_finish_kernel<<<slots / kFinishWarps, kFinishWarps * 32, 0, st>>>(a, slots, d_nbrs, d_dist, uint32_t(row_begin), redo,
                                                                          &counters->redo);
        knn_redo_kernel<U16, QUADS><<<sms, kRedoWarps * 32, 0, st>>>(rows, uint32_t(n), k, a.K, bound, redo, &counters->redo, d_nbrs, d_dist, uint32_t(row_begin),
                                                                        a.choice);
        h->launches += 3;
        CPB_CUDA(cudaGetLastError());
    }
    return 0;
}

}  // namespace

// Plain K-component codes of up to 64 components (four steps of 64 values: a half of the rows has 32 columns of tensor memory).
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
