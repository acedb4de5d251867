#include "resident_ctas.h"

#include <map>
#include <mutex>
#include <tuple>

namespace msda {

cudaError_t resident_ctas(const void* kernel, int threads, size_t smem, int* per_sm) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    struct Key {
        const void* kernel;
        size_t smem;
        int threads, dev;
        bool operator<(const Key& o) const {
            return std::tie(kernel, smem, threads, dev) < std::tie(o.kernel, o.smem, o.threads, o.dev);
        }
    };
    static std::mutex lock;
    static std::map<Key, int> known;   // a handful of entries: kernels x their shared-memory sizes
    const Key key{kernel, smem, threads, dev};
    // Held to the end: the limit only ever grows, because launches of the kernel with more shared
    // memory may be under way and their size is not looked at again. A thread that read the limit
    // before another raised it would lower it.
    std::lock_guard<std::mutex> hold(lock);
    const auto it = known.find(key);
    if (it != known.end()) {
        *per_sm = it->second;
        return cudaSuccess;
    }
    cudaFuncAttributes attr;
    e = cudaFuncGetAttributes(&attr, kernel);
    if (e != cudaSuccess) return e;
    if (smem > static_cast<size_t>(attr.maxDynamicSharedSizeBytes)) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return e;
    }
    int n = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem);
    if (e != cudaSuccess) return e;
    *per_sm = known[key] = n < 1 ? 1 : n;
    return cudaSuccess;
}

}  // namespace msda
