// Device staging memory (staging.h).
#include "staging.h"

#include <mutex>
#include <vector>

namespace lvbgs {

cudaError_t staging_alloc(int device, void** out, size_t bytes, cudaStream_t st) {
    static std::mutex mu;
    static std::vector<cudaMemPool_t> pools;  // by device
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> lk(mu);
        if (device < 0) return cudaErrorInvalidDevice;
        if ((size_t)device >= pools.size()) pools.resize((size_t)device + 1, nullptr);
        if (!pools[device]) {
            cudaMemPoolProps props = {};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = device;
            cudaError_t e = cudaMemPoolCreate(&pools[device], &props);
            if (e != cudaSuccess) {
                pools[device] = nullptr;
                return e;
            }
            unsigned long long keep = kStagingKeep;
            if ((e = cudaMemPoolSetAttribute(pools[device], cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess) {
                cudaMemPoolDestroy(pools[device]);
                pools[device] = nullptr;
                return e;
            }
        }
        pool = pools[device];
    }
    return cudaMallocFromPoolAsync(out, bytes, pool, st);
}

}  // namespace lvbgs
