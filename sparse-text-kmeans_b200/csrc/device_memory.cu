// Device memory kept between the buffers of a process's handles, and the per-kernel attributes that need setting once.
#include <map>
#include <set>
#include <utility>

#include "common.cuh"

namespace cpb {

namespace {

// most bytes kept per device while handles are alive / once the last one is gone
constexpr size_t kKeepAlive = size_t(1) << 30;
constexpr size_t kKeepIdle = size_t(384) << 20;
constexpr int kMaxDevices = 64;

struct Pool {
    std::mutex mu;
    std::multimap<size_t, void*> blocks;  // by size
    size_t kept = 0;
    int handles = 0;

    // returns the largest blocks until at most `most` bytes are kept (mu held)
    void trim(size_t most) {
        while (kept > most && !blocks.empty()) {
            auto it = std::prev(blocks.end());
            kept -= it->first;
            cudaFree(it->second);
            blocks.erase(it);
        }
    }
};
Pool* pools() {
    static Pool* p = new Pool[kMaxDevices];  // (never destroyed: buffers of static handles may outlive every other static)
    return p;
}
thread_local int quiet_depth = 0;

}  // namespace

int device_alloc(void** p, size_t* bytes, int* device, bool* room) {
    CPB_CUDA(cudaGetDevice(device));
    const size_t n = (*bytes + 511) & ~size_t(511);
    if (*device < kMaxDevices) {
        Pool& pool = pools()[*device];
        std::lock_guard<std::mutex> lock(pool.mu);
        // the smallest block that fits, unless it would waste more than a quarter (64 KB for small ones)
        auto it = pool.blocks.lower_bound(n);
        if (it != pool.blocks.end() && it->first <= n + (n / 4 > 65536 ? n / 4 : 65536)) {
            *p = it->second;
            *bytes = it->first;
            pool.kept -= it->first;
            pool.blocks.erase(it);
            return 0;
        }
    }
    cudaError_t e = cudaMalloc(p, n);
    if (e == cudaErrorMemoryAllocation && *device < kMaxDevices) {
        cudaGetLastError();
        Pool& pool = pools()[*device];
        std::lock_guard<std::mutex> lock(pool.mu);
        pool.trim(0);
        e = cudaMalloc(p, n);
    }
    if (e == cudaErrorMemoryAllocation && room) {
        cudaGetLastError();  // the caller goes on without
        *room = false;
        *p = nullptr;
        *bytes = 0;
        return 0;
    }
    CPB_CUDA(e);
    *bytes = n;
    return 0;
}

int reserve_workspace(const cphnsw_b200_index* h, DevBuf& buf, size_t bytes) {
    if (h->workspace_limit && bytes > h->workspace_limit) return kNoRoom;
    bool room = true;
    CPB_TRY(buf.reserve(bytes, &room));
    return room ? 0 : kNoRoom;
}

void device_free(void* p, size_t bytes, int device) {
    int before = 0;
    cudaGetDevice(&before);
    if (before != device) cudaSetDevice(device);
    // nothing that was launched may still use the block when another buffer takes it
    const bool idle = quiet_depth > 0 || cudaDeviceSynchronize() == cudaSuccess;
    bool keep = false;
    if (idle && device < kMaxDevices) {
        Pool& pool = pools()[device];
        std::lock_guard<std::mutex> lock(pool.mu);
        const size_t most = pool.handles ? kKeepAlive : kKeepIdle;
        if (bytes <= most) {
            pool.trim(most - bytes);
            pool.blocks.emplace(bytes, p);
            pool.kept += bytes;
            keep = true;
        }
    }
    if (!keep) cudaFree(p);
    if (before != device) cudaSetDevice(before);
}

void device_handle_created(int device) {
    if (device >= kMaxDevices) return;
    Pool& pool = pools()[device];
    std::lock_guard<std::mutex> lock(pool.mu);
    ++pool.handles;
}

void device_handle_destroyed(int device) {
    if (device >= kMaxDevices) return;
    Pool& pool = pools()[device];
    std::lock_guard<std::mutex> lock(pool.mu);
    if (--pool.handles <= 0) pool.trim(kKeepIdle);
}

int device_release_kept(int device) {
    if (device >= kMaxDevices) return 0;
    int before = 0;
    CPB_CUDA(cudaGetDevice(&before));
    CPB_CUDA(cudaSetDevice(device));
    {
        Pool& pool = pools()[device];
        std::lock_guard<std::mutex> lock(pool.mu);
        pool.trim(0);  // (no kernel uses a kept block: they came in idle)
    }
    CPB_CUDA(cudaSetDevice(before));
    return 0;
}

QuietDevice::QuietDevice() {
    // (a device that reports an error is not quiet: its blocks then go back to the driver)
    if (quiet_depth > 0 || cudaDeviceSynchronize() == cudaSuccess) ++quiet_depth;
    else quiet_depth -= 1 << 20;
}
QuietDevice::~QuietDevice() {
    if (quiet_depth < 0) quiet_depth += 1 << 20;
    else --quiet_depth;
}

cudaError_t allow_max_dynamic_smem_of(const void* kernel) {
    static std::mutex mu;
    static std::set<std::pair<const void*, int>> done;
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    if (done.count({kernel, dev})) return cudaSuccess;
    cudaFuncAttributes fa;
    if ((e = cudaFuncGetAttributes(&fa, kernel)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - int(fa.sharedSizeBytes))) != cudaSuccess) return e;
    done.insert({kernel, dev});
    return cudaSuccess;
}

}  // namespace cpb
