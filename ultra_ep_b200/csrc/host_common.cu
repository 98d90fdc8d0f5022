// Error reporting shared by every C-ABI entry point: integer return codes plus a
// thread-local message (no exceptions cross the ABI).
#include <algorithm>
#include <cstdio>
#include <mutex>
#include <string>

#include "internal.h"
#include "smem_grants.h"

namespace uep {
namespace {
thread_local std::string g_last_error;
}
void set_error(const std::string& msg) { g_last_error = msg; }
int fail(int code, const std::string& msg) {
    g_last_error = msg;
    return code;
}
int fail_cuda(cudaError_t e, const char* what) {
    g_last_error = std::string("CUDA error ") + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ") in " + what;
    return UEP_ERR_CUDA;
}

// SM count of the current device (asked once per device; 0 if the device cannot be queried).
int device_sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess) cached[dev] = n;
    }
    return cached[dev];
}

// Remembered, because each setting costs about as much as a launch.
cudaError_t allow_smem(const void* fn, size_t bytes, bool largest_carveout) {
    if (bytes <= SmemGrants::kDefault && !largest_carveout) return cudaSuccess;
    static std::mutex mu;
    static SmemGrants grants;
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    const size_t have = grants.granted(fn, dev);
    if (have >= std::max(bytes, SmemGrants::kDefault)) return cudaSuccess;
    if (have == 0 && largest_carveout) {
        e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
    }
    if (bytes > SmemGrants::kDefault) {
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
        if (e != cudaSuccess) return e;
    }
    grants.grant(fn, dev, std::max(bytes, SmemGrants::kDefault));
    return cudaSuccess;
}
}  // namespace uep

extern "C" {
const char* uep_last_error(void) { return uep::g_last_error.c_str(); }
const char* uep_version(void) { return "uep_b200 0.1 (sm_100a)"; }
}
