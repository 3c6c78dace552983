// Pieces of the two kernels that sweep operand tiles through the tensor cores (knn_mma.cu, exact_mma.cu): shared-memory
// descriptors, issue and commit, waits; and the split of the exact search's tiles between blocks.
#pragma once

#include "knn_common.cuh"

namespace cpb {
namespace mma {

using knn::kFull;
using knn::smem_u32;

constexpr int kMmaRows = 256;         // rows per block and candidates per tile
constexpr uint32_t kTmemCols = 512;   // all of an SM's; each kernel says what lies where

__device__ __forceinline__ uint64_t operand_desc(uint32_t smem_addr) {
    // K-major, no swizzle: core matrices of 8 rows x 16 bytes, 128 bytes apart along the rows (stride offset) and
    // 256 * 16 bytes apart along K (leading offset); version 1
    uint64_t d = (smem_addr >> 4) & 0x3fffu;
    d |= uint64_t((kMmaRows * 16) >> 4) << 16;
    d |= uint64_t(128 >> 4) << 32;
    d |= uint64_t(1) << 46;
    return d;
}
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r;
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// A bounded wait that also ends when another role of the block has given up.  A poll may sleep for a microsecond: warps
// that spin take the issue slots of those that work.
__device__ __forceinline__ bool mbar_try_wait_us(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, uint32_t limit, volatile int* aborted) {
    for (uint32_t i = 0; i < limit; ++i) {
        if (mbar_try_wait_us(bar, parity)) return true;
        if ((i & 15) == 15 && *aborted) return false;
    }
    return false;
}

// ---- work split -----------------------------------------------------------------------------------------------------
// A launch takes `rts` row tiles against all `cts` candidate tiles: rts * cts steps in row-major order, an equal run of
// them for every block.  When rts is a multiple of the blocks a block takes whole row tiles, and all blocks read the same
// candidate tiles at the same time; otherwise a row tile may be shared by blocks.
struct Split {
    uint64_t steps;
    uint32_t cts, blocks;
    __host__ __device__ uint64_t first_step(uint32_t block) const { return uint64_t(block) * steps / blocks; }
};

}  // namespace mma
}  // namespace cpb
