// Beam search, one warp per query, several expansions per step: same algorithm and same results as search_kernel
// (search.cu) for adjacency rows of up to 32 links.
//
// What bounds a walk is its chain of dependent steps: select the closest unexpanded member of W, read its links, ask
// which are new, fetch and score their codes, rank them into W.  The next member to expand is the next unexpanded one
// unless this expansion admitted something closer, which is rare (3 % of the steps on 1M clustered vectors at beam
// 500).  A step therefore takes the first kRows unexpanded members of W at once: their rows are looked up together,
// their new neighbours are scored together, and then the longest prefix of the rows is committed that the sequential
// walk would have expanded in this order: row t is left for the next step when a neighbour of an earlier row is
// closer than member t.  Candidates are ordered by the total order (distance, id), so W after the committed rows does
// not depend on the order in which their neighbours are admitted, and a row that was not committed has left no trace.
//
// Visited nodes.  W itself decides what is admitted: a node seen before is either a member of W (found there by its
// key when it is ranked) or was turned away or pushed out by members that are closer, and would be again, since the
// worst member of a full W only gets closer.  Remembering visited nodes only saves the scoring, so a filter that may
// forget is enough: 16-bit tags in shared memory, 4 to a bucket (one 64-bit read), the tag and the bucket together
// being a bijection of the id, so that a hit is never wrong.  When the caller asks for statistics (the number of
// distance evaluations counts every node once) or the index is too large for exact tags, the exact set is kept
// instead: one byte per node and slot in global memory holding the number of the slot's last query that visited it.
//
// W is one sorted array of 64-bit keys (ordered distance bits, id, expanded flag) in shared memory.  A step's
// admitted candidates are merged in one pass from the highest position down: the final positions of the candidates
// are marked in a bit set (one word per lane), and the member that moves to position j is the one at j minus the
// marks below it.
//
// The exact rerank (-<q,x> of the best rerank_k, replacing GPUBruteForce::rerank, src/cuda/gpu_encoder.cu:605-664) is
// a kernel of its own, one block per query: inside the walk a single warp would have to read all the vectors.
#include "search_common.cuh"

namespace cpb {
namespace {

using namespace srch;

constexpr int kRows = 4;          // members of W taken per step
constexpr int kBucketLog2 = 9;    // tag filter: 512 buckets of 4 tags = 4 KB per query
constexpr uint32_t kTagBytes = (1u << kBucketLog2) * 8;
constexpr uint64_t kTagNodes = uint64_t(0xffff) << kBucketLog2;  // ids below this have exact tags
constexpr uint64_t kFiller = ~0ull;
constexpr double kOrderReads = 2e9;
constexpr int kOrderSeeds = 8, kOrderLog2 = 12, kOrderBins = 1 << kOrderLog2;
constexpr int kScanKeep = 128;    // most seeds the entry-scan kernel keeps per query: 32 in each of one or four registers a lane
constexpr int kScanWarps = 8;
// Warps (queries) per SM.  A step is about 900 instructions with a chain of memory and shuffle latencies between them,
// so what counts is how many walks an SM has in flight: the query table (16 KB) is therefore read in place, through L1
// and L2, and not held in shared memory, where 7 to 9 walks would fit (1M x 128, 10,000 queries: 5.9 ms with the tables
// in shared memory, 4.3 ms in place with 16 walks per SM, 3.4 ms with 24; 28 at 64 registers: 3.5 ms).
constexpr int kWalkWarps = 24;
constexpr int kFewRanked = 4;     // up to this many candidates are ranked by the whole warp, one after the other

// metrics: asymmetric CP score (kAsym128: its most frequent shape, one-byte codes of 32 rotations at padded dim 128, as
// compile-time facts), symmetric code distance on whole components / on packed sign bits
enum { kAsym = 0, kAsym128 = 1, kSymBytes = 2, kSymPacked = 3 };

struct WalkArgs {
    SearchArgs s;
    const uint64_t* seeds;  // [nq][seed_slots] keys of the entry scan's best, ascending (nullptr: scanned by the walk itself)
    uint32_t seed_slots;
    uint32_t* cand;         // [nq][rerank_k] ids handed to the rerank kernel (nullptr: no rerank)
    const uint32_t* order;  // [nq] the order in which queries are walked and reranked (nullptr: as given)
    uint32_t smem_per_warp;
    uint32_t wcap_slots;    // slots of W's array (multiple of 32)
    int exact_visited;      // bytes in global memory instead of the tag filter
};

__device__ __forceinline__ uint32_t float_order(float d) {
    const uint32_t u = __float_as_uint(d);
    return u ^ (uint32_t(int32_t(u) >> 31) | 0x80000000u);
}
__device__ __forceinline__ float float_unorder(uint32_t u) {
    return __uint_as_float(u ^ ((u & 0x80000000u) ? 0x80000000u : 0xffffffffu));
}
// key of an unexpanded member; bit 0 is the expanded flag
__device__ __forceinline__ uint64_t make_key(float d, uint32_t id) { return (uint64_t(float_order(d)) << 32) | (id << 1); }
__device__ __forceinline__ uint32_t key_id(uint64_t k) { return uint32_t(k) >> 1; }

// ---- tag filter -----------------------------------------------------------------------------------------
// The low bits of an id name its bucket, the high bits plus one are its tag (zero: an empty place).
__device__ __forceinline__ uint32_t tag_of(uint32_t id) { return (id >> kBucketLog2) + 1u; }
__device__ __forceinline__ uint32_t bucket_of(uint32_t id) { return id & ((1u << kBucketLog2) - 1u); }
// flags the halfwords of w that are zero; the lowest flag set is always that of a zero halfword
__device__ __forceinline__ uint32_t zero_half(uint32_t w) { return (w - 0x00010001u) & ~w & 0x80008000u; }

__device__ __forceinline__ bool tag_seen(const uint2* tags, uint32_t id) {
    const uint2 b = tags[bucket_of(id)];
    const uint32_t p = tag_of(id) * 0x00010001u;
    return (zero_half(b.x ^ p) | zero_half(b.y ^ p)) != 0u;
}
// first empty place of the bucket, or a victim; two lanes that meet in one place lose one of the tags
__device__ __forceinline__ void tag_store(uint2* tags, uint32_t id) {
    const uint2 b = tags[bucket_of(id)];
    const uint32_t tag = tag_of(id), z0 = zero_half(b.x), z1 = zero_half(b.y);
    uint32_t pos = tag & 3u;
    if (z0) pos = (z0 & 0x8000u) ? 0u : 1u;
    else if (z1) pos = (z1 & 0x8000u) ? 2u : 3u;
    reinterpret_cast<uint16_t*>(tags + bucket_of(id))[pos] = uint16_t(tag);
}

// ---- W -----------------------------------------------------------------------------------------------------
// Members of W below `key` (binary search, every lane its own key); flags do not matter: a candidate's flag is 0.
// (An eight-ary search, three rounds for 512 members, has the shorter chain of reads but issues 60 instructions a
// round, and was slower: 2,040 against 1,020 cycles where ten lanes search at once.)
__device__ __forceinline__ uint32_t lower_bound(const uint64_t* W, uint32_t count, uint64_t key) {
    uint32_t lo = 0, len = count;
    while (len) {
        const uint32_t half = len >> 1;
        const bool right = W[lo + half] < key;
        lo = right ? lo + half + 1 : lo;
        len = right ? len - half - 1 : half;
    }
    return lo;
}

// Members of W below a key known to every lane: two rounds of a 32-ary search (beams up to 1,024; more passes of 32 in
// the second round beyond).
__device__ __forceinline__ uint32_t lower_bound_warp(const uint64_t* W, uint32_t count, uint64_t key, int lane) {
    if (count == 0) return 0;
    const uint32_t stride = (count + 31) >> 5;
    const uint32_t last = min(count, (uint32_t(lane) + 1) * stride) - 1;  // last member of this lane's block
    const bool less = uint32_t(lane) * stride < count && W[last] < key;
    const uint32_t base = __popc(__ballot_sync(kFull, less)) * stride;    // the blocks entirely below
    if (base >= count) return count;
    uint32_t inside = 0;
    for (uint32_t o = 0; o < stride; o += 32) {
        const uint32_t j = base + o + lane;
        inside += __popc(__ballot_sync(kFull, o + lane < stride && j < count && W[min(j, count - 1)] < key));
    }
    return base + inside;
}

// Scratch of the merge, per warp: the step's keys and, for every 32 positions of W, {marks, marks before}.
// Merges the keys of the lanes in `m` (distinct, none of them in W, rank p = members below the key) into W, which
// keeps the `cap` best.  Returns the lowest position taken.
template <int WORDS>
__device__ __forceinline__ uint32_t merge_into(uint64_t* W, uint32_t& count, uint32_t cap, uint32_t m, uint64_t key, uint32_t p,
                                               uint64_t* kbuf, uint2* marks, int lane) {
    const bool mine = (m >> lane) & 1u;
    const int k = __popc(m);
    const uint32_t newcount = min(cap, count + uint32_t(k));
    constexpr int G = 8;  // chunks of 32 positions moved at a time, highest first: all reads of a group precede its writes
    if (k == 1) {         // one candidate: everything from its position on moves up by one
        const int src = __ffs(m) - 1;
        const uint32_t f = __shfl_sync(kFull, p, src);
        for (int c = int((newcount + 31) >> 5) - 1; c >= int(f >> 5); c -= G) {
            uint64_t e[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int j = (c - g) * 32 + lane;
                e[g] = 0;
                if (j > int(f) && j < int(newcount)) e[g] = W[j - 1];
            }
            __syncwarp();
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int j = (c - g) * 32 + lane;
                if (j > int(f) && j < int(newcount)) W[j] = e[g];
            }
            __syncwarp();
        }
        if (mine) W[f] = key;
        count = newcount;
        __syncwarp();
        return f;
    }
    if (mine) kbuf[__popc(m & ((1u << lane) - 1u))] = key;
#pragma unroll
    for (int w = 0; w < WORDS; ++w) marks[w * 32 + lane].x = 0;
    __syncwarp();
    uint32_t o = 0;  // candidates of the step below this one
    for (int i = 0; i < k; ++i) o += kbuf[i] < key;
    const uint32_t f = p + o;  // final position
    if (mine && (f >> 5) < uint32_t(WORDS * 32)) atomicOr(&marks[f >> 5].x, 1u << (f & 31));
    const uint32_t fmin = __reduce_min_sync(kFull, mine ? f : 0xffffffffu);
    __syncwarp();
    uint32_t carry = 0;
#pragma unroll
    for (int w = 0; w < WORDS; ++w) {
        const uint32_t own = __popc(marks[w * 32 + lane].x);
        uint32_t x = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, x, d);
            if (lane >= d) x += y;
        }
        marks[w * 32 + lane].y = carry + x - own;
        if (WORDS > 1) carry += __shfl_sync(kFull, x, 31);
    }
    __syncwarp();
    for (int c = int((newcount + 31) >> 5) - 1; c >= int(fmin >> 5); c -= G) {
        uint64_t e[G];
        bool move[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int cc = max(c - g, 0);
            const uint2 t = marks[cc];
            const uint32_t j = uint32_t(cc) * 32 + lane;
            move[g] = c - g >= 0 && j >= fmin && j < newcount && !((t.x >> lane) & 1u);
            e[g] = 0;
            if (move[g]) e[g] = W[j - t.y - __popc(t.x & ((1u << lane) - 1u))];
        }
        __syncwarp();
#pragma unroll
        for (int g = 0; g < G; ++g)
            if (move[g]) W[uint32_t(c - g) * 32 + lane] = e[g];
        __syncwarp();
    }
    if (mine && f < cap) W[f] = key;
    count = newcount;
    __syncwarp();
    return fmin;
}

// ---- scoring -------------------------------------------------------------------------------------------------
// Distances of the nodes ids[0, total) (total <= 32) under the asymmetric metric; lane c receives that of node c.
// Four lanes share a node: lane part owns rotations part + 4 i, so the tree's first three levels (16, 8 and 4 apart)
// stay in the lane and the last two are shuffles.  Eight nodes take 8 lookups a lane, against 32 for a lane alone
// (most steps bring fewer than eight) and 13 dependent stages for a warp that shares each node.
template <bool U16, bool FIXED /* one-byte codes, K = 32, P = 128 */>
__device__ __forceinline__ float score_asym(const float* table, const unsigned char* codes, int K_, int P_, const uint32_t* ids, int total,
                                            int lane) {
    const int K = FIXED ? 32 : K_, P = FIXED ? 128 : P_;
    const int row_bytes = K * (U16 ? 2 : 1);
    // (more than eight, as on data without clusters: a lane scores a node, all of them in one pass and 32 lookups of a rotation
    // on its own lines; 100k points of the unit sphere, K = 32, 10,000 queries, beam 500: 16.5 ms in passes of eight, 8.2 so,
    // and 300k clustered ones 3.36 and 3.16)
    if (total > 8) return lane < total ? asym_distance_lane<U16>(table, codes, ids[lane], K, P) : 0.0f;
    float mine = 0.0f;
    const int part = lane & 3;
    const bool vec = FIXED || (row_bytes & 15) == 0;
    const float* part_table = table + part * P;
    for (int g = 0; g < total; g += 8) {
        const uint32_t id = ids[min(g + (lane >> 2), total - 1)];
        const unsigned char* row = codes + size_t(id) * row_bytes;
        float acc = 0.0f;
        for (int c0 = 0; c0 < K; c0 += 32) {
            uint32_t comp[8];
            if (vec && c0 + 32 <= K) {
                constexpr int WORDS = U16 ? 16 : 8;
                const uint4* r4 = reinterpret_cast<const uint4*>(row + c0 * (U16 ? 2 : 1));
                uint32_t x[WORDS];
#pragma unroll
                for (int i = 0; i < WORDS / 4; ++i) {
                    const uint4 v = __ldg(r4 + i);
                    x[4 * i] = v.x, x[4 * i + 1] = v.y, x[4 * i + 2] = v.z, x[4 * i + 3] = v.w;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (U16) comp[i] = ((part & 2) ? x[2 * i + 1] : x[2 * i]) >> (16 * (part & 1)) & 0xffffu;
                    else comp[i] = __byte_perm(x[i], 0u, 0x4440u | uint32_t(part));
                }
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = c0 + part + 4 * i;
                    comp[i] = r < K ? load_component<U16>(row, r) : 0u;
                }
            }
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = c0 + part + 4 * i;
                v[i] = 0.0f;
                if (FIXED || r < K)
                    v[i] = __uint_as_float(__float_as_uint(__ldg(part_table + (c0 + 4 * i) * P + (comp[i] >> 1))) ^ (comp[i] << 31));
            }
#pragma unroll
            for (int h = 4; h >= 1; h >>= 1) {
#pragma unroll
                for (int i = 0; i < h; ++i) v[i] = __fadd_rn(v[i], v[i + h]);
            }
            float t = v[0];
            t = __fadd_rn(t, __shfl_xor_sync(kFull, t, 2));
            t = __fadd_rn(t, __shfl_xor_sync(kFull, t, 1));
            acc = __fadd_rn(acc, t);
        }
        const float d = __shfl_sync(kFull, -acc, ((lane - g) & 7) * 4);
        if (lane >= g && lane < g + 8) mine = d;
    }
    return mine;
}

// ---- entry scan ------------------------------------------------------------------------------------------------
// The n_seed best entry nodes of every query (n_seed <= 128), QG queries per block, the entries dealt to its warps in
// batches of 32, one entry per lane.  Every query reads every entry node, so the scan is bound by table lookups:
// n_entry * K per query, 4 bytes of shared-memory bandwidth each.
//   * The tables of the block's queries are interleaved [block of 32 rotations][index][rotation][query]: one address
//     and one 16-byte read serve four queries.
//   * At step j lane l looks up rotation j XOR l of its entry, so the lanes of a read sit in different banks; the
//     entries' codes are stored with the components in that order (gather_entry_codes).  The balanced tree pairs
//     rotations 16, 8, 4, 2, 1 apart, which differ in one bit of their number, and the XOR leaves it so: the sums keep
//     their bits.
//   * Each warp keeps its 32 best per query, one per lane, or its 128 best, four per lane.  A candidate has to beat the warp's own n_seed-th and the
//     largest of all warps' (n_seed / warps)-th distances, below which n_seed entries are known to lie, so the warps
//     admit about as little as one list would.
struct ScanArgs {
    const float* tables;          // asymmetric: [nq][K][P]
    const unsigned char* qcodes;  // symmetric: [nq][row_bytes]
    const unsigned char* entry_scan;  // asymmetric: rotated codes [n_entry][nblk * 32]; symmetric: code rows / packed words
    const uint32_t* entry;
    uint32_t n_entry, n_seed, nq;
    int K, P, row_bytes, packed_words, resid_kp, resid_mul;
    uint64_t* seeds;  // [nq][32 * KEEP]
    uint32_t* near;   // [nq] the smallest node among the nearest kOrderSeeds (nullptr: not wanted)
};

// compare-exchange across lanes s apart: the lane keeps the smaller key when `low`
__device__ __forceinline__ uint64_t keep_order(uint64_t x, int s, bool low) {
    const uint64_t z = __shfl_xor_sync(kFull, x, s);
    return (z < x) == low ? z : x;
}
// the smallest of an ascending list (32 a register) and of 32 ascending keys, ascending: the smaller and the larger of
// (own, other reversed) are bitonic sequences, the larger go on to the next register
template <int KEEP>
__device__ __forceinline__ void join_sorted(uint64_t (&x)[KEEP], uint64_t other, int lane) {
#pragma unroll
    for (int s = 0; s < KEEP; ++s) {
        const uint64_t y = __shfl_sync(kFull, other, 31 - lane);
        uint64_t lo = y < x[s] ? y : x[s], hi = y < x[s] ? x[s] : y;
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) {
            lo = keep_order(lo, d, (lane & d) == 0);
            if (s + 1 < KEEP) hi = keep_order(hi, d, (lane & d) == 0);
        }
        x[s] = lo;
        other = hi;
    }
}
// the key of rank r
template <int KEEP>
__device__ __forceinline__ uint64_t ranked(const uint64_t (&x)[KEEP], int r) {
    uint64_t k = 0;
#pragma unroll
    for (int s = 0; s < KEEP; ++s) {
        const uint64_t v = __shfl_sync(kFull, x[s], r & 31);
        if (s == r >> 5) k = v;
    }
    return k;
}
constexpr int kSortAdmit = 8;  // from here on sorting a batch (120 instructions) costs less than inserting one by one (14 each)

template <int QG>
struct Vals {
    float v[QG];
};

// two fp32 additions by one instruction, each rounded as the scalar one
__device__ __forceinline__ void add_pair(float& a0, float& a1, float b0, float b1) {
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "+f"(a0), "+f"(a1)
        : "f"(b0), "f"(b1));
}

// S(step, j) of the tree over rotations j ^ lane; w: the entry's components in that order.  (The tree pairs rotations that
// differ in one bit of their number, which the XOR leaves so.)  The scan is bound by its instructions: the address of a
// value is one shift, one mask-and-or and the XOR of lane and j, the sums of two queries are one addition.
template <bool U16, int QG, int STEP, int J>
__device__ __forceinline__ Vals<QG> scan_tree(const unsigned char* table, const uint32_t (&w)[U16 ? 16 : 8], uint32_t lane_at,
                                              uint32_t row_mask) {
    Vals<QG> r;
    if constexpr (STEP == 32) {
        constexpr int PER = U16 ? 2 : 4, BITS = U16 ? 16 : 8;
        constexpr int SH = (J % PER) * BITS;                      // the component's position in its word
        constexpr int UP = QG == 4 ? 8 : (QG == 2 ? 7 : 6);       // twice an index to the bytes of its row of the table
        const uint32_t word = w[J / PER];
        const uint32_t sign = word << (31 - SH);
        const uint32_t row = UP >= SH ? word << (UP >= SH ? UP - SH : 0) : word >> (UP >= SH ? 0 : SH - UP);
        const uint32_t at = (row & row_mask) | (lane_at ^ uint32_t(J * QG * 4));  // the mask keeps it inside the table
        float x[QG];
        if constexpr (QG == 4) {
            const float4 f = *reinterpret_cast<const float4*>(table + at);
            x[0] = f.x, x[1] = f.y, x[2] = f.z, x[3] = f.w;
        } else if constexpr (QG == 2) {
            const float2 f = *reinterpret_cast<const float2*>(table + at);
            x[0] = f.x, x[1] = f.y;
        } else {
            x[0] = *reinterpret_cast<const float*>(table + at);
        }
#pragma unroll
        for (int i = 0; i < QG; ++i) r.v[i] = __uint_as_float(__float_as_uint(x[i]) ^ (sign & 0x80000000u));
    } else {
        r = scan_tree<U16, QG, STEP * 2, J>(table, w, lane_at, row_mask);
        const Vals<QG> b = scan_tree<U16, QG, STEP * 2, J + STEP>(table, w, lane_at, row_mask);
        if constexpr (QG == 1) {
            r.v[0] = __fadd_rn(r.v[0], b.v[0]);
        } else {
#pragma unroll
            for (int i = 0; i < QG; i += 2) add_pair(r.v[i], r.v[i + 1], b.v[i], b.v[i + 1]);
        }
    }
    return r;
}

template <bool U16, int METRIC, int QG, int KEEP>
__global__ void __launch_bounds__(kScanWarps * 32, KEEP == 1 ? 3 : 2)
entry_scan_kernel(ScanArgs a) {
    extern __shared__ __align__(16) unsigned char scan_smem[];
    __shared__ uint64_t lists[kScanWarps][QG][32 * KEEP];
    __shared__ uint32_t bound[QG][kScanWarps];  // ordered distance of each warp's (n_seed / warps)-th best
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t q0 = blockIdx.x * QG;
    const int nblk = (a.K + 31) / 32;
    if (threadIdx.x < QG * kScanWarps) bound[threadIdx.x / kScanWarps][threadIdx.x % kScanWarps] = 0xffffffffu;
    if constexpr (METRIC == kAsym) {
        // lane = rotation; four indices of QG queries per pass
        float* tab = reinterpret_cast<float*>(scan_smem);
        const int quads = a.P / 4;
        for (int u = warp; u < nblk * quads; u += kScanWarps) {
            const int blk = u / quads, i4 = (u % quads) * 4, r = blk * 32 + lane;
            float x[QG][4];
#pragma unroll
            for (int g = 0; g < QG; ++g) {
                float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < a.K && q0 + g < a.nq)
                    f = __ldg(reinterpret_cast<const float4*>(a.tables + (size_t(q0 + g) * a.K + r) * a.P + i4));
                x[g][0] = f.x, x[g][1] = f.y, x[g][2] = f.z, x[g][3] = f.w;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float* dst = tab + ((size_t(blk) * a.P + i4 + i) * 32 + lane) * QG;
                if constexpr (QG == 4) *reinterpret_cast<float4*>(dst) = make_float4(x[0][i], x[1][i], x[2][i], x[3][i]);
                else if constexpr (QG == 2) *reinterpret_cast<float2*>(dst) = make_float2(x[0][i], x[1][i]);
                else *dst = x[0][i];
            }
        }
    } else {  // the queries' codes, as bytes or packed sign bits
        for (int g = 0; g < QG; ++g) {
            const unsigned char* src = a.qcodes + size_t(min(q0 + g, a.nq - 1)) * a.row_bytes;
            if (METRIC == kSymBytes) {
                for (int i = threadIdx.x; i < a.row_bytes; i += kScanWarps * 32) scan_smem[size_t(g) * ((a.row_bytes + 15) / 16 * 16) + i] = src[i];
            } else if (warp == 0) {
                for (int i = 0; i < a.packed_words; ++i) {
                    const int r = 32 * i + lane;
                    const uint32_t word = __ballot_sync(kFull, r < a.K && (src[r * (U16 ? 2 : 1)] & 1u));
                    if (lane == 0) reinterpret_cast<uint32_t*>(scan_smem)[g * a.packed_words + i] = word;
                }
            }
        }
    }
    __syncthreads();

    uint64_t best[QG][KEEP];
    uint32_t thr[QG];  // ordered distance a candidate must not exceed
#pragma unroll
    for (int g = 0; g < QG; ++g) {
        thr[g] = 0xffffffffu;
#pragma unroll
        for (int s = 0; s < KEEP; ++s) best[g][s] = kFiller;
    }
    const int pub = (int(a.n_seed) + kScanWarps - 1) / kScanWarps - 1;
    for (uint32_t e0 = warp * 32; e0 < a.n_entry; e0 += kScanWarps * 32) {
        const uint32_t e = e0 + lane;
        const bool ok = e < a.n_entry;
        const uint32_t ee = ok ? e : a.n_entry - 1;
        const uint32_t id = __ldg(a.entry + ee);
        float d[QG];
        if constexpr (METRIC == kAsym) {
            constexpr int WORDS = U16 ? 16 : 8;
            const uint4* row = reinterpret_cast<const uint4*>(a.entry_scan + size_t(ee) * nblk * (U16 ? 64 : 32));
#pragma unroll
            for (int g = 0; g < QG; ++g) d[g] = 0.0f;
            for (int blk = 0; blk < nblk; ++blk) {
                uint32_t w[WORDS];
#pragma unroll
                for (int i = 0; i < WORDS / 4; ++i) {
                    const uint4 v = __ldg(row + blk * (WORDS / 4) + i);
                    w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
                }
                const Vals<QG> s = scan_tree<U16, QG, 1, 0>(scan_smem + size_t(blk) * a.P * 32 * QG * 4, w, uint32_t(lane * QG * 4),
                                                               uint32_t(2 * a.P - 2) << (QG == 4 ? 8 : (QG == 2 ? 7 : 6)));
#pragma unroll
                for (int g = 0; g < QG; ++g) d[g] = __fadd_rn(d[g], s.v[g]);
            }
#pragma unroll
            for (int g = 0; g < QG; ++g) d[g] = -d[g];
        } else if (METRIC == kSymBytes && (a.row_bytes & 15) == 0 && !a.resid_mul) {
            // an entry's code is read once for all queries of the block
            uint32_t differ[QG];
#pragma unroll
            for (int g = 0; g < QG; ++g) differ[g] = 0;
            const uint4* row = reinterpret_cast<const uint4*>(a.entry_scan + size_t(ee) * a.row_bytes);
            const uint4* codes = reinterpret_cast<const uint4*>(scan_smem);  // a row apart
            for (int w = 0; w < a.row_bytes / 16; ++w) {
                const uint4 x = __ldg(row + w);
#pragma unroll
                for (int g = 0; g < QG; ++g) {
                    const uint4 c = codes[g * (a.row_bytes / 16) + w];
                    differ[g] += quad_mismatches<U16>(x, c.x, c.y, c.z, c.w);
                }
            }
#pragma unroll
            for (int g = 0; g < QG; ++g) d[g] = float(differ[g]);
        } else {
#pragma unroll
            for (int g = 0; g < QG; ++g) {
                if (METRIC == kSymPacked)
                    d[g] = packed_distance_lane(reinterpret_cast<const uint32_t*>(scan_smem) + g * a.packed_words,
                                                reinterpret_cast<const uint32_t*>(a.entry_scan), ee, a.packed_words, a.resid_kp, a.resid_mul);
                else
                    d[g] = sym_distance_lane<U16>(scan_smem + size_t(g) * ((a.row_bytes + 15) / 16 * 16), a.entry_scan, ee, a.K, a.resid_kp,
                                                  a.resid_mul);
            }
        }
#pragma unroll
        for (int g = 0; g < QG; ++g) {
            const uint64_t key = make_key(d[g], id);
            const uint32_t others = lane < kScanWarps ? *reinterpret_cast<volatile uint32_t*>(&bound[g][lane]) : 0u;
            const uint32_t lim = min(thr[g], __reduce_max_sync(kFull, others));
            uint32_t m = __ballot_sync(kFull, ok && uint32_t(key >> 32) <= lim);
            if (m == 0) continue;
            if (__popc(m) > kSortAdmit) {  // many: sorted and joined as one list
                uint64_t x = ((m >> lane) & 1u) ? key : kFiller;
#pragma unroll
                for (int k2 = 2; k2 <= 32; k2 <<= 1)
#pragma unroll
                    for (int s = k2 >> 1; s >= 1; s >>= 1) x = keep_order(x, s, ((lane & s) == 0) == ((lane & k2) == 0 || k2 == 32));
                join_sorted(best[g], x, lane);
            } else {
                while (m) {
                    const int src = __ffs(m) - 1;
                    m &= m - 1;
                    const uint64_t k = __shfl_sync(kFull, key, src);
                    int r = 0;
#pragma unroll
                    for (int s = 0; s < KEEP; ++s) r += __popc(__ballot_sync(kFull, best[g][s] < k));
#pragma unroll
                    for (int s = KEEP - 1; s >= 0; --s) {
                        uint64_t up = __shfl_up_sync(kFull, best[g][s], 1);
                        if (s > 0) {
                            const uint64_t carry = __shfl_sync(kFull, best[g][s - 1], 31);
                            if (lane == 0) up = carry;
                        }
                        const int at = 32 * s + lane;
                        best[g][s] = at < r ? best[g][s] : (at == r ? k : up);
                    }
                }
            }
            thr[g] = uint32_t(ranked(best[g], int(a.n_seed) - 1) >> 32);
            if (lane == pub) *reinterpret_cast<volatile uint32_t*>(&bound[g][warp]) = uint32_t(best[g][0] >> 32);
        }
    }
#pragma unroll
    for (int g = 0; g < QG; ++g)
#pragma unroll
        for (int s = 0; s < KEEP; ++s) lists[warp][g][32 * s + lane] = best[g][s];
    __syncthreads();
    // one warp per query joins the sorted lists
    for (int g = warp; g < QG; g += kScanWarps) {
        if (q0 + g >= a.nq) continue;
        uint64_t x[KEEP];
#pragma unroll
        for (int s = 0; s < KEEP; ++s) x[s] = lists[0][g][32 * s + lane];
        for (int o = 1; o < kScanWarps; ++o) {
            for (int s = 0; s < KEEP; ++s) {
                if (KEEP > 1 && lists[o][g][32 * s] >= ranked(x, 32 * KEEP - 1)) break;  // (and so are the ones behind it)
                join_sorted(x, lists[o][g][32 * s + lane], lane);
            }
        }
#pragma unroll
        for (int s = 0; s < KEEP; ++s) a.seeds[size_t(q0 + g) * (32 * KEEP) + 32 * s + lane] = x[s];
        if (a.near) {
            const uint32_t least = __reduce_min_sync(kFull, lane < kOrderSeeds ? key_id(x[0]) : kInvalidNode);
            if (lane == 0) a.near[q0 + g] = least;
        }
    }
}

// ---- order of the queries ------------------------------------------------------------------------------------------
// Queries of one cluster rerank much the same vectors.  Taken one after the other they find them in L2; as given, a base that
// does not fit L2 is read from HBM once for each.  Queries with the same nearest entry node, of whose kOrderSeeds nearest the
// smallest stands for all, go together, in any order otherwise.  One block: a count, a scan and a scatter over kOrderBins bins
// that such nodes are hashed to.  All kernels of a search, with the 10 us of this one, on four seeds in turn: 10,000 queries, 1M x 128,
// 500 reranked 3,002 to 3,011 us as given, 2,895 to 2,917 in order; 2,000 of 960 dimensions, 100k, 1,000 reranked 2,811 to 2,850
// and 2,620 to 2,684.  (By the nearest of one seed 2,954 to 2,990 and 2,723 to 2,757, of two 2,943 to 2,980 and 2,724 to 2,743.)
__global__ void __launch_bounds__(1024) order_queries_kernel(const uint32_t* __restrict__ near, uint32_t nq, uint32_t* __restrict__ order) {
    constexpr int kEach = kOrderBins / 1024;
    __shared__ uint32_t bins[kOrderBins], sums[32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto bin_of = [](uint32_t node) { return node * 2654435761u >> (32 - kOrderLog2); };
#pragma unroll
    for (int i = 0; i < kEach; ++i) bins[tid * kEach + i] = 0;
    __syncthreads();
#pragma unroll 4
    for (uint32_t q = tid; q < nq; q += 1024) atomicAdd(&bins[bin_of(__ldg(near + q))], 1u);
    __syncthreads();
    uint32_t own = 0, at[kEach];
#pragma unroll
    for (int i = 0; i < kEach; ++i) at[i] = own, own += bins[tid * kEach + i];
    auto scan = [&](uint32_t x) {  // inclusive, over the lanes
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, x, d);
            if (lane >= uint32_t(d)) x += y;
        }
        return x;
    };
    const uint32_t upto = scan(own);
    if (lane == 31) sums[warp] = upto;
    __syncthreads();
    if (warp == 0) {
        const uint32_t of = sums[lane];
        sums[lane] = scan(of) - of;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kEach; ++i) bins[tid * kEach + i] = at[i] + upto - own + sums[warp];
    __syncthreads();
#pragma unroll 4
    for (uint32_t q = tid; q < nq; q += 1024) order[atomicAdd(&bins[bin_of(__ldg(near + q))], 1u)] = q;
}

template <bool U16, int METRIC, int WORDS>
__global__ void __launch_bounds__(kWalkWarps * 32) search_walk_kernel(WalkArgs w) {
    extern __shared__ __align__(16) unsigned char walk_smem[];
    const SearchArgs& a = w.s;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    constexpr bool SYM = METRIC == kSymBytes || METRIC == kSymPacked;
    const int row_bytes = a.K * (U16 ? 2 : 1);
    uint64_t* W = reinterpret_cast<uint64_t*>(walk_smem + size_t(w.smem_per_warp) * warp);
    uint2* tags = reinterpret_cast<uint2*>(W + w.wcap_slots);
    uint64_t* kbuf = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(tags) + (w.exact_visited ? 0 : kTagBytes));
    uint2* marks = reinterpret_cast<uint2*>(kbuf + 32);
    uint32_t* cid = reinterpret_cast<uint32_t*>(marks + WORDS * 32);
    uint32_t* front = cid + 32;  // the first unexpanded members of W
    unsigned char* qcode = reinterpret_cast<unsigned char*>(front + 8);  // symmetric metric: code bytes or packed words
    uint32_t* qpacked = reinterpret_cast<uint32_t*>(qcode);

    const uint32_t n = uint32_t(a.n);  // below 2^31
    const uint32_t slot = blockIdx.x * warps + warp;
    uint8_t* vis = w.exact_visited ? a.visited + size_t(slot) * a.vis_stride : nullptr;
    uint32_t epoch = w.exact_visited ? a.epochs[slot] : 0u;

    while (true) {
        uint32_t q = 0;
        if (lane == 0) q = atomicAdd(a.next_query, 1u);
        q = __shfl_sync(kFull, q, 0);
        if (q >= a.nq) break;
        if (w.order) q = __ldg(w.order + q);
        __syncwarp();
        const float* table = SYM ? nullptr : a.tables + size_t(q) * a.K * a.P;
        if (SYM) {
            const unsigned char* src = static_cast<const unsigned char*>(a.qcodes) + size_t(q) * row_bytes;
            if (METRIC == kSymBytes) {
                for (int i = lane; i < row_bytes; i += 32) qcode[i] = src[i];
            } else {
                for (int i = 0; i < a.packed_words; ++i) {
                    const int r = 32 * i + lane;
                    const uint32_t word = __ballot_sync(kFull, r < a.K && (src[r * (U16 ? 2 : 1)] & 1u));
                    if (lane == 0) qpacked[i] = word;
                }
            }
        }
        if (!w.exact_visited) {
            for (int i = lane; i < int(kTagBytes / 16); i += 32) reinterpret_cast<uint4*>(tags)[i] = make_uint4(0u, 0u, 0u, 0u);
        } else if (++epoch == 256) {  // the 8-bit epoch wraps: forget every earlier query
            uint4* v4 = reinterpret_cast<uint4*>(vis);
            for (uint64_t i = lane; i < a.vis_stride / 16; i += 32) v4[i] = make_uint4(0u, 0u, 0u, 0u);
            epoch = 1;
        }
        __syncwarp();

        uint32_t count = 0, cur = 0, nexp = 0, nevals = 0;

        // distance of node `id` of lane `lane` < total (ids also in cid[])
        auto score = [&](int total, uint32_t id) -> float {
            if (METRIC == kSymPacked)
                return lane < total ? packed_distance_lane(qpacked, a.packed, id, a.packed_words, a.resid_kp, a.resid_mul) : 0.0f;
            if (METRIC == kSymBytes)
                return lane < total ? sym_distance_lane<U16>(qcode, a.codes, id, a.K, a.resid_kp, a.resid_mul) : 0.0f;
            return score_asym<U16, METRIC == kAsym128>(table, static_cast<const unsigned char*>(a.codes), a.K, a.P, cid, total, lane);
        };
        auto remember = [&](bool mine, uint32_t id) {
            if (w.exact_visited) {
                if (mine) vis[id] = uint8_t(epoch);
            } else if (mine) {
                tag_store(tags, id);
            }
        };

        // ---- entry nodes (search_engine.hpp:105-115): all of them are offered, or the n_seed best of a scan
        const bool scan = a.n_seed < a.n_entry;
        const uint32_t cap0 = scan ? a.n_seed : a.beam;
        if (w.seeds) {
            for (uint32_t s = lane; s < w.seed_slots; s += 32) {
                const uint64_t k = w.seeds[size_t(q) * w.seed_slots + s];
                const bool have = k != kFiller && s < cap0;
                if (have) W[s] = k;
                count += __popc(__ballot_sync(kFull, have));
            }
            nevals += a.n_entry;
            __syncwarp();
        }
        for (uint32_t e0 = w.seeds ? a.n_entry : 0u; e0 < a.n_entry; e0 += 32) {
            const uint32_t e = e0 + lane;
            const uint32_t id = e < a.n_entry ? __ldg(a.entry + e) : kInvalidNode;
            const bool ok = id < n;
            const uint32_t m = __ballot_sync(kFull, ok);  // (entry ids are distinct and valid up to the end of the list)
            const int total = 32 - __clz(int(m));
            if (total == 0) continue;
            float d;
            if (METRIC == kSymPacked || METRIC == kSymBytes) {
                d = ok ? sym_distance_lane<U16>(METRIC == kSymBytes ? qcode : reinterpret_cast<const unsigned char*>(a.qcodes) + size_t(q) * row_bytes,
                                                a.entry_codes, e, a.K, a.resid_kp, a.resid_mul) : 0.0f;
            } else {
                d = ok ? asym_distance_lane<U16>(table, a.entry_codes, e, a.K, a.P) : 0.0f;
            }
            nevals += __popc(m);
            const uint64_t key = make_key(d, id);
            const bool adm = ok && (count < cap0 || key < W[count - 1]);
            const uint32_t am = __ballot_sync(kFull, adm);
            if (am) merge_into<WORDS>(W, count, cap0, am, key, adm ? lower_bound(W, count, key) : 0u, kbuf, marks, lane);
            if (!scan) remember(ok, id);
        }
        if (scan) {  // the seeds are offered to the walk: marked visited, scored once more (a beam narrower than the
                     // seed set keeps the best `beam` of them)
            nevals += count;
            for (uint32_t p = lane; p < count; p += 32) remember(true, key_id(W[p]));
            if (count > a.beam) count = a.beam;
        }
        __syncwarp();

        // ---- walk
        uint32_t pre_node[kRows], pre_row[kRows];  // links loaded one step ahead for the members expected next
#pragma unroll
        for (int b = 0; b < kRows; ++b) pre_node[b] = kInvalidNode, pre_row[b] = kInvalidNode;
        while (true) {
            // the first kRows unexpanded members of the first window of 32 that has any (search_engine.hpp:121-123)
            uint32_t un = 0;
            while (cur < count) {  // four windows at a time: an admission near the front sends the cursor back to it
                uint32_t u[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t p = cur + 32 * i + lane;
                    u[i] = __ballot_sync(kFull, p < count && !(uint32_t(W[min(p, count - 1)]) & 1u));
                }
                if (u[0] | u[1] | u[2] | u[3]) {
                    const int i = u[0] ? 0 : (u[1] ? 1 : (u[2] ? 2 : 3));
                    un = u[0] ? u[0] : (u[1] ? u[1] : (u[2] ? u[2] : u[3]));
                    cur += 32 * i;
                    break;
                }
                cur += 128;
            }
            if (!un) break;
            const uint32_t below = (1u << lane) - 1u;
            const uint32_t order = __popc(un & below);
            const bool open_member = (un >> lane) & 1u;
            const uint64_t ek = W[min(cur + lane, count - 1)];
            if (open_member && order < 2 * kRows) front[order] = uint32_t(ek) >> 1;
            const uint32_t sel = __ballot_sync(kFull, open_member && order < kRows);  // the members taken
            const int have = __popc(un);
            __syncwarp();
            uint32_t row[kRows], node[kRows];
#pragma unroll
            for (int b = 0; b < kRows; ++b) {
                node[b] = b < have ? front[b] : kInvalidNode;
                row[b] = pre_row[b];
                if (node[b] != pre_node[b])
                    row[b] = (node[b] != kInvalidNode && lane < a.M) ? __ldg(a.adj + size_t(node[b]) * a.M + lane) : kInvalidNode;
            }
            // the members behind them are the next step's unless this one changes the front of W
#pragma unroll
            for (int b = 0; b < kRows; ++b) {
                pre_node[b] = kRows + b < have ? front[kRows + b] : kInvalidNode;
                pre_row[b] = (pre_node[b] != kInvalidNode && lane < a.M) ? __ldg(a.adj + size_t(pre_node[b]) * a.M + lane) : kInvalidNode;
            }
            // neighbours not seen before, row by row
            uint32_t fresh[kRows];
            if (w.exact_visited) {
                uint32_t vb[kRows];
#pragma unroll
                for (int b = 0; b < kRows; ++b) vb[b] = row[b] < n ? uint32_t(__ldcg(vis + row[b])) : epoch;
#pragma unroll
                for (int b = 0; b < kRows; ++b) fresh[b] = __ballot_sync(kFull, vb[b] != epoch);
            } else {
#pragma unroll
                for (int b = 0; b < kRows; ++b)
                    fresh[b] = __ballot_sync(kFull, row[b] < n && !tag_seen(tags, row[b]));
            }
            // as many leading rows as bring at most 32 candidates; lane c owns candidate c
            int total = 0, rows = 0, first_of[kRows];
            bool open = true;
#pragma unroll
            for (int b = 0; b < kRows; ++b) {
                const int nf = __popc(fresh[b]);
                open = open && node[b] != kInvalidNode && total + nf <= 32;
                first_of[b] = total;
                if (open) {
                    if ((fresh[b] >> lane) & 1u) cid[total + __popc(fresh[b] & below)] = row[b];
                    total += nf;
                    ++rows;
                }
            }
            __syncwarp();
            uint32_t commit = uint32_t(rows);
            uint32_t id = kInvalidNode, my_row = 0, p = 0xffffffffu;
            uint64_t key = kFiller;
            bool own = false;
            if (total) {
                own = lane < total;
                id = own ? cid[lane] : kInvalidNode;
#pragma unroll
                for (int b = 1; b < kRows; ++b)
                    if (b < rows && lane >= first_of[b]) my_row = b;
                const float d = score(total, id);
                // a node listed by two rows (or twice in one) belongs to the first
                const uint32_t grp = __match_any_sync(kFull, id);
                own = own && (__ffs(grp) - 1) == lane;
                key = make_key(d, id);
                bool adm = own && (count < a.beam || key < W[count - 1]);
                uint32_t am = __ballot_sync(kFull, adm);
                if (am) {
                    if (__popc(am) <= kFewRanked) {  // the warp ranks one key after the other
                        for (uint32_t r = am; r;) {
                            const int src = __ffs(r) - 1;
                            r &= r - 1;
                            const uint32_t at = lower_bound_warp(W, count, __shfl_sync(kFull, key, src), lane);
                            if (lane == src) p = at;
                        }
                    } else if (adm) {
                        p = lower_bound(W, count, key);
                    }
                    if (adm) {
                        // a forgotten node that is a member of W
                        if (p < count && (W[p] >> 1) == (key >> 1)) adm = false;
                    }
                    if (adm) {
                        // rows t with member t below this candidate stay in order; the row that found it is done by then
                        const uint32_t rel = p - cur;  // cur <= position of every selected member
                        const uint32_t bl = p <= cur ? 0u : (rel >= 32u ? sel : sel & ((1u << rel) - 1u));
                        commit = max(my_row + 1u, uint32_t(__popc(bl)));
                    }
                    commit = min(uint32_t(rows), __reduce_min_sync(kFull, commit));
                    am = __ballot_sync(kFull, adm && my_row < commit);
                }
                own = own && my_row < commit;
                remember(own, id);
                nevals += __popc(__ballot_sync(kFull, own));
                // the committed members carry their flag before positions move
                if (open_member && order < commit) W[cur + lane] = ek | 1u;
                __syncwarp();
                if (am) {
                    const uint32_t f = merge_into<WORDS>(W, count, a.beam, am, key, p, kbuf, marks, lane);
                    cur = min(cur, f);
                }
            } else {
                if (open_member && order < commit) W[cur + lane] = ek | 1u;
                __syncwarp();
            }
            nexp += commit;
        }

        // ---- results: the ids the rerank kernel scores, or the k best with their distances
        if (w.cand) {
            uint32_t* out = w.cand + size_t(q) * a.rerank_k;
            for (uint32_t p = lane; p < a.rerank_k; p += 32) out[p] = p < count ? key_id(W[p]) : kInvalidNode;
        } else {
            for (uint32_t p = lane; p < a.k; p += 32) {
                const uint64_t e = p < count ? W[p] : 0;
                a.out_ids[size_t(q) * a.k + p] = p < count ? key_id(e) : kInvalidNode;
                a.out_dist[size_t(q) * a.k + p] = p < count ? float_unorder(uint32_t(e >> 32)) : INFINITY;
            }
        }
        if (a.stats && lane == 0) {
            a.stats[2 * size_t(q)] = nexp;
            a.stats[2 * size_t(q) + 1] = nevals;
        }
        __syncwarp();
    }
    if (w.exact_visited && lane == 0) a.epochs[slot] = epoch;
}

// ---- few queries: a block per query ----------------------------------------------------------------------------------
// With fewer queries than the chip has room for walks, what counts is the length of one walk: its steps in sequence,
// some 5,000 cycles each for a warp alone.  Here eight warps share a query and a step takes the first 32 unexpanded members of W
// (those of a window of 32), four rows a warp, dealt out in turn (where a row brings so many candidates that a warp has room for
// one only, as on data without clusters, the step still has the first eight); the prefix committed grows from 3.4 rows to 32 where
// the beam is nearly settled, and the rows' lookups and scores run side by side.  Rows, candidates and the committed prefix are
// those of search_walk_kernel, so the results are too.
//
// A step meets at barriers: every warp says which bound its candidates put on the prefix; the candidates of the rows within it
// are listed with their ranks in W; repeats (a node found by two rows) are struck out; those left are ranked among each other and
// go to their places in the other of W's two arrays; and every member moves there by the number of them that rank before it,
// found by bisection.  What bounds it is the chain of round trips, some 6,400 cycles a step: rows, codes and tables from L2, the
// bisection of W, barriers.  One query on 100k x 128, beam 500, all kernels: 302 us with the candidates of all rows listed before
// the prefix was known (a query's first ten or so steps find 100 to 250 and commit one row), ranked by a thread an entry and every
// member held against every entry; 224 with 16 rows a step, 213 with 24, 191 with 32.  Two windows
// and 64 rows: 186, but of the sphere 3 % slower than with 32.  Codes of the rows expected next loaded ahead, W known to be shared
// memory: no faster.
constexpr uint32_t kStruck = 0xffffffffu;  // no place

constexpr int kSquadWarps = 8;
constexpr int kSquadThreads = kSquadWarps * 32;
constexpr int kSquadRows = 4;                            // per warp
constexpr int kSquadFront = kSquadWarps * kSquadRows;    // members of W taken per step
static_assert(kSquadFront == 32, "the unexpanded members of a window");
constexpr size_t kSquadStatic = 6160;                    // its static shared memory

template <bool U16, int METRIC>
__global__ void __launch_bounds__(kSquadThreads, 4) search_squad_kernel(WalkArgs w) {
    extern __shared__ __align__(16) unsigned char walk_smem[];
    __shared__ uint64_t list_key[kSquadThreads];
    __shared__ uint32_t list_place[kSquadThreads];  // members of W below
    // a warp's candidates and front until the step's prefix is known; then, until it ends, the listed keys that are kept
    __shared__ uint64_t kept_key[kSquadThreads];
    static_assert(sizeof(kept_key) == kSquadWarps * (32 + kSquadFront) * 4, "32 candidates and kSquadFront members a warp");
    __shared__ uint32_t sorted_place[kSquadThreads];  // of the entries kept, in order
    __shared__ uint32_t listed, prefix, seeded, kept_all;
    const SearchArgs& a = w.s;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t tid = threadIdx.x, below = (1u << lane) - 1u;
    const uint32_t q = blockIdx.x, n = uint32_t(a.n);
    unsigned char* qcode = walk_smem + size_t(w.wcap_slots) * 16 + kTagBytes;  // symmetric metrics
    uint64_t* W = reinterpret_cast<uint64_t*>(walk_smem);
    uint64_t* W2 = W + w.wcap_slots;
    uint2* tags = reinterpret_cast<uint2*>(W2 + w.wcap_slots);
    uint32_t* cid = reinterpret_cast<uint32_t*>(kept_key) + warp * (32 + kSquadFront);
    uint32_t* front = cid + 32;
    constexpr bool SYM = METRIC == kSymBytes || METRIC == kSymPacked;
    const float* table = SYM ? nullptr : a.tables + size_t(q) * a.K * a.P;
    if (SYM && warp == 0) {  // the query's code, as bytes or packed sign bits
        const int row_bytes = a.K * (U16 ? 2 : 1);
        const unsigned char* src = static_cast<const unsigned char*>(a.qcodes) + size_t(q) * row_bytes;
        if (METRIC == kSymBytes) {
            for (int i = lane; i < row_bytes; i += 32) qcode[i] = src[i];
        } else {
            for (int i = 0; i < a.packed_words; ++i) {
                const int r = 32 * i + lane;
                const uint32_t word = __ballot_sync(kFull, r < a.K && (src[r * (U16 ? 2 : 1)] & 1u));
                if (lane == 0) reinterpret_cast<uint32_t*>(qcode)[i] = word;
            }
        }
    }

    for (uint32_t i = tid; i < kTagBytes / 16; i += kSquadThreads) reinterpret_cast<uint4*>(tags)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0) listed = 0, prefix = kSquadFront;
    __syncthreads();

    auto score = [&](int total, uint32_t id) -> float {
        if (METRIC == kSymPacked)
            return lane < total ? packed_distance_lane(reinterpret_cast<const uint32_t*>(qcode), a.packed, id, a.packed_words, a.resid_kp, a.resid_mul) : 0.0f;
        if (METRIC == kSymBytes) return lane < total ? sym_distance_lane<U16>(qcode, a.codes, id, a.K, a.resid_kp, a.resid_mul) : 0.0f;
        return score_asym<U16, METRIC == kAsym128>(table, static_cast<const unsigned char*>(a.codes), a.K, a.P, cid, total, lane);
    };

    // entry nodes: the scan's best, in order; or all of them (up to 128), 32 a warp
    if (w.seeds) {
        if (warp == 0) {
            uint32_t have = 0;
            for (uint32_t s = lane; s < w.seed_slots; s += 32) {
                const uint64_t k = w.seeds[size_t(q) * w.seed_slots + s];
                const bool seed = k != kFiller && s < a.n_seed;
                if (seed) tag_store(tags, key_id(k));
                if (seed && s < a.beam) W[s] = k;
                have += __popc(__ballot_sync(kFull, seed));
            }
            if (lane == 0) seeded = min(have, a.beam);
        }
    } else {
        uint64_t k = kFiller;
        if (warp * 32 < int(a.n_entry)) {
            const int total = int(min(a.n_entry - warp * 32, 32u));
            const uint32_t id = lane < total ? __ldg(a.entry + tid) : kInvalidNode;
            cid[lane] = id;
            __syncwarp();
            const float d = score(total, id);
            if (lane < total) {
                k = make_key(d, id);
                tag_store(tags, id);
            }
        }
        list_key[tid] = k;
        __syncthreads();
        uint32_t rank = 0;
        for (uint32_t i = 0; i < a.n_entry; ++i) rank += list_key[i] < k;
        if (k != kFiller && rank < a.beam) W[rank] = k;
        if (tid == 0) seeded = min(a.n_entry, a.beam);
    }
    __syncthreads();
    uint32_t count = seeded, cur = 0;

    while (true) {
        // the first unexpanded members of the first window of 32 that has any: every warp finds them for itself
        uint32_t un = 0;
        while (cur < count) {
            uint32_t u[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t p = cur + 32 * i + lane;
                u[i] = __ballot_sync(kFull, p < count && !(uint32_t(W[min(p, count - 1)]) & 1u));
            }
            if (u[0] | u[1] | u[2] | u[3]) {
                const int i = u[0] ? 0 : (u[1] ? 1 : (u[2] ? 2 : 3));
                un = u[0] ? u[0] : (u[1] ? u[1] : (u[2] ? u[2] : u[3]));
                cur += 32 * i;
                break;
            }
            cur += 128;
        }
        if (!un) break;
        const uint32_t order = __popc(un & below);
        const bool open = (un >> lane) & 1u;
        const uint64_t ek = W[min(cur + lane, count - 1)];
        if (open) front[order] = uint32_t(ek) >> 1;
        const int have = __popc(un);
        __syncwarp();
        uint32_t row[kSquadRows], fresh[kSquadRows];
#pragma unroll
        for (int b = 0; b < kSquadRows; ++b) {
            const int t = b * kSquadWarps + warp;
            row[b] = t < have && lane < a.M ? __ldg(a.adj + size_t(front[t]) * a.M + lane) : kInvalidNode;
        }
#pragma unroll
        for (int b = 0; b < kSquadRows; ++b) fresh[b] = __ballot_sync(kFull, row[b] < n && !tag_seen(tags, row[b]));
        // as many of the warp's rows as bring at most 32 candidates
        int total = 0, first_of[kSquadRows];
        uint32_t bound = uint32_t(have);
        bool room = true;
#pragma unroll
        for (int b = 0; b < kSquadRows; ++b) {
            const int nf = __popc(fresh[b]);
            first_of[b] = total;
            if (room && total + nf > 32) {
                room = false;
                bound = min(bound, uint32_t(b * kSquadWarps + warp));
            }
            if (room) {
                if ((fresh[b] >> lane) & 1u) cid[total + __popc(fresh[b] & below)] = row[b];
                total += nf;
            }
        }
        __syncwarp();
        uint32_t id = kInvalidNode, my_row = 0, p = 0;
        uint64_t key = kFiller;
        bool own = false, adm = false;
        if (total) {
            own = lane < total;
            id = own ? cid[lane] : kInvalidNode;
#pragma unroll
            for (int b = 0; b < kSquadRows; ++b)
                if (lane >= first_of[b]) my_row = b * kSquadWarps + warp;
            const float d = score(total, id);
            const uint32_t grp = __match_any_sync(kFull, id);
            own = own && (__ffs(grp) - 1) == lane;
            key = make_key(d, id);
            adm = own && (count < a.beam || key < W[count - 1]);
            if (adm) {
                p = lower_bound(W, count, key);
                if (p < count && (W[p] >> 1) == (key >> 1)) adm = false;  // a forgotten node that is a member of W
            }
            if (adm) {
                const uint32_t rel = p - cur;  // cur <= position of every selected member
                const uint32_t bl = p <= cur ? 0u : (rel >= 32u ? un : un & ((1u << rel) - 1u));
                bound = min(bound, max(my_row + 1u, uint32_t(__popc(bl))));
            }
        }
        bound = __reduce_min_sync(kFull, bound);
        if (lane == 0) atomicMin(&prefix, bound);
        __syncthreads();
        const uint32_t commit = prefix;
        if (own && my_row < commit) tag_store(tags, id);
        adm = adm && my_row < commit;
        const uint32_t am = __ballot_sync(kFull, adm);
        if (am) {
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&listed, uint32_t(__popc(am)));
            at = __shfl_sync(kFull, at, 0) + __popc(am & below);
            if (adm) {
                list_key[at] = key;
                list_place[at] = p;
            }
        }
        __syncthreads();
        const uint32_t m = listed;
        uint32_t kept = 0, lowest = kStruck;
        if (tid == 0) prefix = kSquadFront, kept_all = 0;
        if (m) {
            // several threads an entry, as many as there are; they share the loop over the others
            const int share = m <= 32 ? 3 : (m <= 64 ? 2 : (m <= 128 ? 1 : 0));
            const uint32_t threads = 1u << share, entry = tid >> share, part = tid & (threads - 1);
            const uint32_t mates = (kFull >> (32 - threads)) << (lane & ~(threads - 1));
            const bool have_entry = entry < m;
            const uint64_t mine = have_entry ? list_key[entry] : 0;
            bool twice = false;
            if (have_entry) {
#pragma unroll 4
                for (uint32_t i = part; i < entry; i += threads) twice |= list_key[i] == mine;
            }
            const uint32_t repeats = __ballot_sync(kFull, twice);
            const bool keep = have_entry && !(repeats & mates);
            const uint32_t place = keep ? list_place[entry] : kStruck;
            if (have_entry && part == 0) kept_key[entry] = keep ? mine : kFiller;  // (ranks above all; list_key is still being read)
            __syncthreads();
            if (tid == 0) listed = 0;
            uint32_t rank = 0;
            if (keep) {
#pragma unroll 4
                for (uint32_t i = part; i < m; i += threads) rank += kept_key[i] < mine;
            }
            for (uint32_t d = 1; d < threads; d <<= 1) rank += __shfl_xor_sync(kFull, rank, d);
            const bool first = keep && part == 0;
            const uint32_t kept_here = __popc(__ballot_sync(kFull, first));
            if (lane == 0 && kept_here) atomicAdd(&kept_all, kept_here);
            if (first) {
                sorted_place[rank] = place;
                if (place + rank < a.beam) W2[place + rank] = mine;
            }
            __syncthreads();
            kept = kept_all, lowest = sorted_place[0];
        }
        // the members of the committed rows carry their flag from now on
        const uint32_t flag = __ballot_sync(kFull, open && order < commit);
        if (kept) {
            const uint32_t newcount = min(a.beam, count + kept);
            for (uint32_t j = tid; j < count; j += kSquadThreads) {
                uint64_t e = W[j];
                const uint32_t rel = j - cur;
                if (j >= cur && rel < 32u && ((flag >> rel) & 1u)) e |= 1u;
                uint32_t up = 0, end = j < lowest ? 0u : kept;  // the entries placed at j or before
                while (up < end) {
                    const uint32_t mid = (up + end) >> 1;
                    if (sorted_place[mid] <= j) up = mid + 1;
                    else end = mid;
                }
                if (j + up < newcount) W2[j + up] = e;
            }
            uint64_t* t = W;
            W = W2;
            W2 = t;
            count = newcount;
        } else if (warp == 0 && ((flag >> lane) & 1u)) {
            W[cur + lane] = ek | 1u;
        }
        cur = min(cur, lowest);
        __syncthreads();
    }

    if (w.cand) {
        uint32_t* out = w.cand + size_t(q) * a.rerank_k;
        for (uint32_t p = tid; p < a.rerank_k; p += kSquadThreads) out[p] = p < count ? key_id(W[p]) : kInvalidNode;
    } else {
        for (uint32_t p = tid; p < a.k; p += kSquadThreads) {
            const uint64_t e = p < count ? W[p] : 0;
            a.out_ids[size_t(q) * a.k + p] = p < count ? key_id(e) : kInvalidNode;
            a.out_dist[size_t(q) * a.k + p] = p < count ? float_unorder(uint32_t(e >> 32)) : INFINITY;
        }
    }
}

// ---- exact rerank: one block per query -------------------------------------------------------------------------
// 8 lanes per candidate row (128-bit loads), 32 rows of a block in flight per pass; the dot product is accumulated
// with fmaf per lane and folded 4, 2, 1, as the fused rerank of search_kernel does.  The keys are then sorted in
// shared memory and the k best written out.
// (256 threads a block; 1,024 when there are few queries: 28 against 11 us for one query with 500 candidates)
template <int kRerankThreads>
__global__ void __launch_bounds__(kRerankThreads)
search_rerank_kernel(const float* __restrict__ vectors, const float* __restrict__ queries, const uint32_t* __restrict__ cand,
                     const uint32_t* __restrict__ order /* or nullptr */, uint32_t rr, uint32_t slots /* power of two >= rr */, int dim, uint32_t k, uint32_t* __restrict__ out_ids,
                     float* __restrict__ out_dist) {
    extern __shared__ __align__(16) unsigned char rr_smem[];
    uint64_t* keys = reinterpret_cast<uint64_t*>(rr_smem);
    float* qsm = reinterpret_cast<float*>(keys + slots);
    const size_t q = order ? __ldg(order + blockIdx.x) : blockIdx.x;
    const uint32_t* ids = cand + q * rr;
    for (int i = threadIdx.x; i < dim; i += kRerankThreads) qsm[i] = __ldg(queries + q * dim + i);
    __syncthreads();
    const int g = threadIdx.x >> 3, j = threadIdx.x & 7;
    const bool vec4 = (dim & 3) == 0;
#pragma unroll 4
    for (uint32_t c0 = 0; c0 < slots; c0 += kRerankThreads / 8) {
        const uint32_t c = c0 + g;
        const uint32_t id = c < rr ? __ldg(ids + c) : kInvalidNode;
        float acc = 0.0f;
        if (id != kInvalidNode) {
            const float* x = vectors + size_t(id) * dim;
            if (vec4) {
                for (int i = 4 * j; i < dim; i += 32) {
                    const float4 xv = __ldg(reinterpret_cast<const float4*>(x + i));
                    const float4 qv = *reinterpret_cast<const float4*>(qsm + i);
                    acc = fmaf(xv.x, qv.x, acc);
                    acc = fmaf(xv.y, qv.y, acc);
                    acc = fmaf(xv.z, qv.z, acc);
                    acc = fmaf(xv.w, qv.w, acc);
                }
            } else {
                for (int i = j; i < dim; i += 8) acc = fmaf(__ldg(x + i), qsm[i], acc);
            }
        }
        acc += __shfl_xor_sync(kFull, acc, 4);
        acc += __shfl_xor_sync(kFull, acc, 2);
        acc += __shfl_xor_sync(kFull, acc, 1);
        if (j == 0 && c < slots) keys[c] = id != kInvalidNode ? make_key(-acc, id) : kFiller;
    }
    __syncthreads();
    for (uint32_t k2 = 2; k2 <= slots; k2 <<= 1) {
        for (uint32_t jj = k2 >> 1; jj > 0; jj >>= 1) {
            for (uint32_t t = threadIdx.x; t < slots / 2; t += kRerankThreads) {
                const uint32_t lo = ((t & ~(jj - 1)) << 1) | (t & (jj - 1)), hi = lo | jj;
                const uint64_t x = keys[lo], y = keys[hi];
                if ((y < x) == ((lo & k2) == 0)) {
                    keys[lo] = y;
                    keys[hi] = x;
                }
            }
            __syncthreads();
        }
    }
    for (uint32_t p = threadIdx.x; p < k; p += kRerankThreads) {
        const uint64_t e = p < slots ? keys[p] : kFiller;
        out_ids[q * k + p] = e != kFiller ? key_id(e) : kInvalidNode;
        out_dist[q * k + p] = e != kFiller ? float_unorder(uint32_t(e >> 32)) : INFINITY;
    }
}

template <bool U16, int METRIC, int QG>
int launch_scan_t(cphnsw_b200_index* h, const ScanArgs& a, size_t smem, cudaStream_t st) {
    auto go = [&](auto kernel) -> int {
        CPB_CUDA(allow_max_dynamic_smem(kernel));
        kernel<<<(a.nq + QG - 1) / QG, kScanWarps * 32, smem, st>>>(a);
        return 0;
    };
    if (a.n_seed <= 32) CPB_TRY(go(entry_scan_kernel<U16, METRIC, QG, 1>));
    else CPB_TRY(go(entry_scan_kernel<U16, METRIC, QG, 4>));
    h->launches++;
    CPB_CUDA(cudaGetLastError());
    return 0;
}

template <bool U16>
int launch_scan(cphnsw_b200_index* h, const ScanArgs& a, int metric, cudaStream_t st) {
    const size_t row = (size_t(a.row_bytes) + 15) / 16 * 16;
    // several queries share a block's reads of the entry codes once every SM has a block of its own
    const bool many = a.nq > uint32_t(h->sm_count);
    if (metric == kSymBytes)
        return many ? launch_scan_t<U16, kSymBytes, 4>(h, a, 4 * row, st) : launch_scan_t<U16, kSymBytes, 1>(h, a, row, st);
    if (metric == kSymPacked)
        return many ? launch_scan_t<U16, kSymPacked, 4>(h, a, size_t(16) * a.packed_words, st)
                    : launch_scan_t<U16, kSymPacked, 1>(h, a, size_t(4) * a.packed_words, st);
    const size_t table = size_t((a.K + 31) / 32) * 32 * a.P * 4;
    if (many && a.nq > 2 * uint32_t(h->sm_count) && 4 * table <= 72 * 1024) return launch_scan_t<U16, kAsym, 4>(h, a, 4 * table, st);
    if (many && 2 * table <= 72 * 1024) return launch_scan_t<U16, kAsym, 2>(h, a, 2 * table, st);
    return launch_scan_t<U16, kAsym, 1>(h, a, table, st);
}

template <bool U16, int METRIC>
int launch_walk_t(cphnsw_b200_index* h, const WalkArgs& w, int blocks, int warps, cudaStream_t st) {
    const size_t smem = size_t(w.smem_per_warp) * warps;
    auto go = [&](auto kernel) -> int {
        CPB_CUDA(allow_max_dynamic_smem(kernel));
        kernel<<<unsigned(blocks), unsigned(warps) * 32, smem, st>>>(w);
        return 0;
    };
    if (w.wcap_slots <= 1024) return go(search_walk_kernel<U16, METRIC, 1>);
    return go(search_walk_kernel<U16, METRIC, 4>);  // beams up to 4,096: four words of the merge's bit set per lane
}

template <bool U16, int METRIC>
int launch_squad_t(const WalkArgs& w, size_t smem, cudaStream_t st) {
    CPB_CUDA(allow_max_dynamic_smem(search_squad_kernel<U16, METRIC>));
    search_squad_kernel<U16, METRIC><<<w.s.nq, kSquadThreads, smem, st>>>(w);
    return 0;
}

}  // namespace

// Fills in the launch shape and runs walk and rerank.  a.next_query is zero on entry.
int launch_search_walk(cphnsw_b200_index* h, SearchCtx& cx, SearchArgs a, bool sym, cudaStream_t st) {
    WalkArgs w;
    w.s = a;
    w.cand = nullptr;
    w.order = nullptr;
    if (a.rerank_k) {
        CPB_TRY(cx.d_cand.reserve(size_t(a.nq) * a.rerank_k * 4 + 16));
        w.cand = cx.d_cand.as<uint32_t>();
    }
    uint32_t top = a.beam > a.n_seed ? a.beam : a.n_seed;
    w.wcap_slots = (top + 31) & ~31u;
    w.exact_visited = (a.stats != nullptr || a.n > kTagNodes) ? 1 : 0;
    if (w.exact_visited) {
        CPB_TRY(prepare_search_scratch(h, cx, st));
        w.s.visited = cx.d_visited.as<uint8_t>();
        w.s.vis_stride = cx.vis_stride;
        w.s.epochs = cx.d_epochs.as<uint32_t>();
    }
    const bool u16 = a.comp_bytes == 2;
    const int metric = sym ? (a.packed ? kSymPacked : kSymBytes) : (!u16 && a.K == 32 && a.P == 128 ? kAsym128 : kAsym);
    const size_t row = (size_t(a.K) * a.comp_bytes + 15) / 16 * 16;
    const size_t words = w.wcap_slots <= 1024 ? 1 : 4;
    // W, tags, merge scratch (keys, marks), candidate ids, front, the query's code
    w.smem_per_warp = uint32_t((size_t(w.wcap_slots) * 8 + (w.exact_visited ? 0 : kTagBytes) + 256 + words * 256 + 128 + 32 +
                                (sym ? row : 0) + 15) / 16 * 16);
    int warps = int((226 * 1024) / w.smem_per_warp);
    // Visited arrays: 16 per SM.  Query tables above 32 KB: with 24 walks an SM those in flight (227 MB at 64 KB) leave L2 where
    // the walks read all of them, as on data without clusters (100k x 300, K = 32, 10,000 queries, beam 500: 58.7 ms with 24,
    // 41.2 with 16; 960-d |N|: 59.2 and 39.5); clustered data, which read little of them, lose 3 to 12 % (4.40 and 4.94, 6.89 and
    // 7.10 ms).  At 32 KB clustered data
    // would lose 20 % (4.14 and 5.02 ms, K = 64), and the others keep up as they are (33.9 ms, 40.4 with two warps per query).
    const bool wide_table = !sym && size_t(a.K) * a.P * 4 > 32 * 1024;
    const int most = (w.exact_visited || wide_table) && warps > 16 ? 16 : kWalkWarps;
    if (warps > most) warps = most;
    const int per_sm = int((a.nq + h->sm_count - 1) / h->sm_count);  // a small batch spreads over all SMs
    if (warps > per_sm) warps = per_sm;
    if (warps < 1) warps = 1;
    if (!cx.wide) warps = 1;
    const uint64_t want = (uint64_t(a.nq) + warps - 1) / warps;
    const int blocks = int(want < uint64_t(h->sm_count) ? want : uint64_t(h->sm_count));
    w.seeds = nullptr;
    w.seed_slots = 0;
    const size_t scan_table = size_t((a.K + 31) / 32) * 32 * a.P * 4;
    if (a.n_seed < a.n_entry && a.n_seed <= uint32_t(kScanKeep) && (sym || (a.P >= 4 && scan_table <= 200 * 1024))) {
        ScanArgs sc;
        sc.tables = a.tables;
        sc.qcodes = static_cast<const unsigned char*>(a.qcodes);
        sc.entry_scan = metric == kSymBytes ? static_cast<const unsigned char*>(a.entry_codes) : h->d_entry_scan.as<unsigned char>();
        sc.entry = a.entry;
        sc.n_entry = a.n_entry;
        sc.n_seed = a.n_seed;
        sc.nq = a.nq;
        sc.K = a.K;
        sc.P = a.P;
        sc.row_bytes = a.K * a.comp_bytes;
        sc.packed_words = a.packed_words;
        sc.resid_kp = a.resid_kp;
        sc.resid_mul = a.resid_mul;
        w.seed_slots = a.n_seed <= 32 ? 32 : kScanKeep;
        CPB_TRY(cx.d_seeds.reserve(size_t(a.nq) * (w.seed_slots * 8 + 8)));
        sc.seeds = cx.d_seeds.as<uint64_t>();
        w.seeds = sc.seeds;
        // The order costs 10 us.  It is of use where links, codes and vectors do not fit L2, and made up for where the queries read them
        // many times.  Four seeds, us as given and in order: 10,000 queries on 1M x 128, 3.4 GB, 3,002 to 3,011 and 2,895 to 2,917; on
        // 300k x 128 2,515 to 2,543 and 2,468 to 2,493; 2,000 on 100k x 960, 8 GB, 2,811 to 2,850 and 2,620 to 2,684; on 100k x 512,
        // 2.2 GB, 1,168 to 1,174 and 1,131 to 1,140; 600 on 100k x 960, 2.4 GB, 1,787 to 1,834 and 1,791 to 1,818, where it breaks even.
        sc.near = nullptr;
        const double node_bytes = double(a.M) * 4 + double(row), vector_bytes = a.rerank_k ? double(a.dim) * 4 : 0.0;
        if (a.nq > 2 * uint32_t(h->sm_count) && double(a.n) * (node_bytes + vector_bytes) > double(h->l2_bytes) &&
            double(a.nq) * (a.beam * node_bytes + a.rerank_k * vector_bytes) > kOrderReads) {
            sc.near = reinterpret_cast<uint32_t*>(sc.seeds + size_t(a.nq) * w.seed_slots);
        }
        CPB_TRY(a.comp_bytes == 2 ? launch_scan<true>(h, sc, metric, st) : launch_scan<false>(h, sc, metric, st));
        if (sc.near) {
            order_queries_kernel<<<1, 1024, 0, st>>>(sc.near, a.nq, sc.near + a.nq);
            h->launches++;
            w.order = sc.near + a.nq;
        }
    }
    // Few queries: a block each.  Against a warp each, us for 1 / 148 / 296 / 592 queries: 100k x 128, beam 500, K = 32 166 / 212 /
    // 284 / 341 against 475 / 507 / 530 / 563; K = 64, a table of 32 KB, 237 / 309 / 364 / 509 against 845 / 914 / 956 / 980; 60k
    // points of the sphere, K = 32 1,139 / 1,308 / 1,453 / 1,875 against 1,815 at 592; sign-bit codes, K = 64, beam 200, 164 / 203 /
    // 233 / 278 against 244 / 289 / 350 / 359, of the sphere 339 / 453 / 497 / 592 against 565 / 604 / 629 / 640; code distance, K =
    // 32, of the sphere 425 / 530 / 575 / 704 against 601 / 698 / 709 / 758.
    //   How many an SM: four run at once where shared memory has room for their beams, to some 2,950, else three, and the others go in
    // a second wave.  Query tables of 32 KB and more: four, in waves or not (beam 4,096, 592 queries: 0.78 of a warp each).  Symmetric
    // metrics: four, in waves up to 499 queries (sign bits, K = 64, beam 4,096: 0.98 of a warp each at 500, 1.10 at 592).  Small
    // tables, whose warps are nearly as fast, 445 and 555 queries, of a warp each: K = 32, M = 32, beam 100 0.86 and 0.96, beam 40
    // 0.93 and 1.04, up to 444 0.76 to 0.94; M = 24, beam 64 0.94 and 0.98; beam 4,096 1.13 and 1.36, of the sphere 1.27 and 1.34, up
    // to 444 0.51 to 0.81.  Rows of 16 links bring few candidates a step: beam 40 1.06 at 333, 1.17 at 555, of the sphere 1.03 and
    // 1.13; beam 200 0.79 and 0.94, of the sphere 1.04 and 1.25.  More than four an SM: 800 queries 486 us against 613 on clusters,
    // but 2,945 against 1,897 of the sphere.
    const size_t squad_smem = size_t(w.wcap_slots) * 16 + kTagBytes + (sym ? row : 0);
    const bool four = size_t(228 * 1024) / (squad_smem + kSquadStatic + 1024) >= 4;
    uint32_t eighths = 32;  // of a query an SM
    if (sym) eighths = four ? 32 : 27;
    else if (size_t(a.K) * a.P * 4 < 32 * 1024) eighths = a.M <= 16 ? (a.beam < 200 ? 16 : 24) : (a.beam < 64 || !four ? 24 : 30);
    const uint32_t squads = uint32_t(h->sm_count) * eighths / 8;
    if (!w.exact_visited && a.nq <= squads && (w.seeds || (a.n_seed >= a.n_entry && a.n_entry <= 128))) {
#define CPB_SQUAD(X) (u16 ? launch_squad_t<true, X>(w, squad_smem, st) : launch_squad_t<false, X>(w, squad_smem, st))
        switch (metric) {
            case kAsym: CPB_TRY(CPB_SQUAD(kAsym)); break;
            case kAsym128: CPB_TRY((launch_squad_t<false, kAsym128>(w, squad_smem, st))); break;
            case kSymBytes: CPB_TRY(CPB_SQUAD(kSymBytes)); break;
            default: CPB_TRY(CPB_SQUAD(kSymPacked)); break;
        }
#undef CPB_SQUAD
    } else {
#define CPB_WALK(X) (u16 ? launch_walk_t<true, X>(h, w, blocks, warps, st) : launch_walk_t<false, X>(h, w, blocks, warps, st))
    switch (metric) {
        case kAsym: CPB_TRY(CPB_WALK(kAsym)); break;
        case kAsym128: CPB_TRY((launch_walk_t<false, kAsym128>(h, w, blocks, warps, st))); break;
        case kSymBytes: CPB_TRY(CPB_WALK(kSymBytes)); break;
        default: CPB_TRY(CPB_WALK(kSymPacked)); break;
    }
#undef CPB_WALK
    }
    h->launches++;
    CPB_CUDA(cudaGetLastError());
    if (a.rerank_k) {
        uint32_t slots = 32;
        while (slots < a.rerank_k) slots <<= 1;
        const size_t smem = size_t(slots) * 8 + (size_t(a.dim) * 4 + 15) / 16 * 16;
        if (a.nq <= uint32_t(2 * h->sm_count)) {
            CPB_CUDA(allow_max_dynamic_smem(search_rerank_kernel<1024>));
            search_rerank_kernel<1024><<<a.nq, 1024, smem, st>>>(a.vectors, a.queries, w.cand, w.order, a.rerank_k, slots, a.dim, a.k, a.out_ids,
                                                                a.out_dist);
        } else {
            CPB_CUDA(allow_max_dynamic_smem(search_rerank_kernel<256>));
            search_rerank_kernel<256><<<a.nq, 256, smem, st>>>(a.vectors, a.queries, w.cand, w.order, a.rerank_k, slots, a.dim, a.k, a.out_ids,
                                                              a.out_dist);
        }
        h->launches++;
        CPB_CUDA(cudaGetLastError());
    }
    return 0;
}

}  // namespace cpb
