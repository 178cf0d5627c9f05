// pool.cu -- device memory of the handles, their workspaces and the tile
// build's temporaries, from one private stream-ordered pool per device.
//
// A handle is some 45 arrays.  Mapping each one anew cost more than building
// it: 40 x 8 MB took 57 ms to cudaMalloc and 14 ms to cudaFree on one B200, and
// the default pool returns its memory at every synchronisation, so the scans'
// temporaries were mapped again on each call.  From this pool an allocation
// takes 2 us.  A 96^3 build with one product took 33 ms, of which 1 ms was
// kernels.
//
// What the pool holds beyond live allocations is bounded: at most kKeepBytes
// (the release threshold follows what is live, see follow(); more goes back at
// the next synchronisation), and once nothing is live, at most what was live
// since it was last empty (mf_pool_settle).  A failed allocation gives the rest back and tries again.
// The pool is stream-ordered and safe with any number of threads.
//
// A handle's memory is given back the way cudaFree would, which the rest of a
// program may rely on: all work on the device has ended by then, and another
// thread's stream capture survives it.  cudaDeviceSynchronize and any call on the
// legacy stream next to a captured blocking stream invalidate captures, so the wait
// is the one inside cudaFree (mf_device_wait), and arrays go back with cudaFree,
// which for pool memory neither waits nor ties the block to a stream (freed on a
// stream, each was reused through an event: 55 us more a build).
#include "mf_internal.cuh"

#include <mutex>

namespace {

constexpr int kMaxDevices = 64;
constexpr unsigned long long kKeepBytes = 1ull << 30;

struct DevicePool {
    cudaMemPool_t pool;
    void *keep;                 // holds the small-allocation block that mf_device_wait uses
};
std::mutex g_mu;
DevicePool g_pool[kMaxDevices];

// The current device's pool, made on first use.
int pool_of(int dev, DevicePool *out)
{
    if (dev < 0 || dev >= kMaxDevices) return MF_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_pool[dev].pool) {
        cudaMemPoolProps pr = {};
        pr.allocType = cudaMemAllocationTypePinned;
        pr.location.type = cudaMemLocationTypeDevice;
        pr.location.id = dev;
        cudaMemPool_t p = nullptr;
        MF_CUDA_TRY(cudaMemPoolCreate(&p, &pr));
        unsigned long long keep = kKeepBytes;
        void *block = nullptr;
        cudaError_t e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);   // nothing live yet
        if (e == cudaSuccess) e = cudaMalloc(&block, 1);
        if (e != cudaSuccess) {
            cudaMemPoolDestroy(p);
            MF_CUDA_TRY(e);
        }
        g_pool[dev] = {p, block};
    }
    *out = g_pool[dev];
    return MF_SUCCESS;
}

// The driver compares the release threshold with all the memory a pool holds,
// live allocations included.  With a fixed one, handles above it (three 128^3
// systems) had every freed array unmapped at the next synchronisation and mapped
// again for the next solve (first solve of a handle 4.9 -> 8.5 ms).
void follow(cudaMemPool_t pool)
{
    unsigned long long used = 0;
    if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess) {
        used += kKeepBytes;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &used);
    }
    cudaGetLastError();
}

constexpr size_t kFollowBytes = 4u << 20;    // allocations that move the threshold

}  // namespace

int mf_pool_alloc(void **p, size_t bytes, cudaStream_t s)
{
    *p = nullptr;
    int dev = 0;
    MF_CUDA_TRY(cudaGetDevice(&dev));
    DevicePool dp;
    const int rc = pool_of(dev, &dp);
    if (rc != MF_SUCCESS) return rc;
    cudaMemPool_t pool = dp.pool;
    cudaError_t e = cudaMallocFromPoolAsync(p, bytes > 0 ? bytes : 1, pool, s);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        mf_device_wait();
        if (cudaMemPoolTrimTo(pool, 0) == cudaSuccess)
            e = cudaMallocFromPoolAsync(p, bytes > 0 ? bytes : 1, pool, s);
    }
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
    }
    MF_CUDA_TRY(e);
    if (bytes >= kFollowBytes) follow(pool);
    return MF_SUCCESS;
}

void mf_pool_free(void *p, cudaStream_t s)
{
    if (p && cudaFreeAsync(p, s) != cudaSuccess) cudaGetLastError();
}

// cudaFree of an allocation of cudaMalloc waits for the whole device.
void mf_device_wait()
{
    void *p = nullptr;
    if (cudaMalloc(&p, 1) == cudaSuccess) cudaFree(p);
    else cudaDeviceSynchronize();
    cudaGetLastError();
}

void mf_pool_give_back(void *const *p, int count)
{
    for (int k = 0; k < count; k++)
        if (p[k] && cudaFree(p[k]) != cudaSuccess) cudaGetLastError();
}

void mf_pool_settle(int dev)
{
    DevicePool dp;
    unsigned long long used = 0, high = 0, held = 0, zero = 0;
    if (pool_of(dev, &dp) != MF_SUCCESS) return;
    cudaMemPool_t pool = dp.pool;
    follow(pool);
    if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess || used > 0 ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemHigh, &high) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    if (held > high) cudaMemPoolTrimTo(pool, (size_t)high);
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrUsedMemHigh, &zero);
    cudaGetLastError();
}

MfDeviceGuard::MfDeviceGuard(int dev) : old(-1)
{
    int cur = -1;
    if (cudaGetDevice(&cur) == cudaSuccess && cur != dev && cudaSetDevice(dev) == cudaSuccess) old = cur;
}

MfDeviceGuard::~MfDeviceGuard()
{
    if (old >= 0) cudaSetDevice(old);
}
