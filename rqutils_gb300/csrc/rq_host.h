// Host-side helpers shared by the entry points: error reporting, CUDA checks, launch sizing,
// scratch layout.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "rqsqd.h"

#define RQ_API extern "C" __attribute__((visibility("default")))

namespace rq {

// Thread-local last error message (rq_last_error).
void set_error(const std::string &msg);
int fail(int code, const std::string &msg);

// Returns RQ_E_CUDA with a message if `e` is an error.
int cuda_fail(cudaError_t e, const char *what);

#define RQ_CUDA(call)                                                 \
    do {                                                              \
        cudaError_t e_ = (call);                                      \
        if (e_ != cudaSuccess) return ::rq::cuda_fail(e_, #call);     \
    } while (0)

#define RQ_TRY(call)                                                  \
    do {                                                              \
        int rc_ = (call);                                             \
        if (rc_ != RQ_OK) return rc_;                                 \
    } while (0)

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

// Number of SMs of the current device (cached per device).
int sm_count();

// Scratch layout (bytes from the scratch base):
//   [0, 16)         reserved
//   [16, 32)        device error flag (int32)
//   [32, 32 + R)    grid-reduction area (its counter, then the partials), R = reduce_scratch_bytes()
//   [.., ..)        scan block sums for D rows (int64)
constexpr size_t kScratchErr = 16;
constexpr size_t kScratchReduce = 32;
size_t scratch_scan_offset();
size_t scratch_bytes(int64_t D);

inline int *scratch_err(void *scratch) {
    return reinterpret_cast<int *>(static_cast<char *>(scratch) + kScratchErr);
}
inline void *scratch_reduce(void *scratch) {
    return static_cast<char *>(scratch) + kScratchReduce;
}
inline int64_t *scratch_scan(void *scratch) {
    return reinterpret_cast<int64_t *>(static_cast<char *>(scratch) + scratch_scan_offset());
}

int vtype_size(int32_t vtype);

// Launch settings of one kernel: whether it has been opted into dynamic shared memory and its
// occupancy at one shared-memory size.  Each launcher keeps one entry per host thread and device
// (cache_slot), so threads never share an entry and devices with different SM counts never see each
// other's occupancy.
struct KernelLaunchCache {
    bool opted = false;
    size_t occ_smem = ~size_t(0);
    int occ_blocks = 1;
};
constexpr int kMaxCachedDevices = 64;

// Opt kern into all the dynamic shared memory that the current device allows beside its static part.  The
// runtime keeps one limit per kernel and device for all threads, and a later call can lower it, so every
// call sets the same one: a thread's launch never depends on what another has asked for since.  (The
// limit is no allocation; the launch's own size decides the occupancy.)
template <typename KernT>
int opt_into_shared(KernT kern, KernelLaunchCache &c) {
    if (c.opted) return RQ_OK;
    cudaFuncAttributes a{};
    int dev = 0, most = 0;
    RQ_CUDA(cudaFuncGetAttributes(&a, kern));
    RQ_CUDA(cudaGetDevice(&dev));
    RQ_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    RQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)a.sharedSizeBytes));
    c.opted = true;
    return RQ_OK;
}

// The same, and kern's resident blocks per SM at `block` threads and smem bytes of dynamic shared memory,
// querying the runtime only when `c` does not hold the answer yet (the occupancy query is also reached
// while a stream is being captured, where only stream work should be issued).
template <typename KernT>
int configure_kernel(KernT kern, KernelLaunchCache &c, size_t smem, int block, int *per_sm) {
    RQ_TRY(opt_into_shared(kern, c));
    if (c.occ_smem != smem) {
        int per = 0;
        RQ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, block, smem));
        c.occ_blocks = per < 1 ? 1 : per;
        c.occ_smem = smem;
    }
    *per_sm = c.occ_blocks;
    return RQ_OK;
}

// This thread's entry for the current device in a launcher's table.
inline int cache_slot(KernelLaunchCache (&table)[kMaxCachedDevices], KernelLaunchCache **out) {
    int dev = 0;
    RQ_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxCachedDevices) return fail(RQ_E_RANGE, "device index out of range");
    *out = &table[dev];
    return RQ_OK;
}

}  // namespace rq
