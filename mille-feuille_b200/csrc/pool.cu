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
// the next synchronisation and when a handle is destroyed), and once nothing is
// live, at most what was live since it was last empty (mf_pool_settle).  A failed
// allocation gives the rest back and tries again.
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

#include <memory>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace {

constexpr int kMaxDevices = 64;
constexpr unsigned long long kKeepBytes = 1ull << 30;

// One pool per device and context: a cudaDeviceReset ends the context's pool, and
// the next handle makes another (the entries of ended contexts stay).
struct DevicePool {
    int dev;
    MfContext ctx;
    cudaMemPool_t pool;
    void *keep;                      // holds the small-allocation block that mf_device_wait uses
    unsigned long long live, high;   // bytes allocated now, and at most since none were
};
struct Allocation {
    DevicePool *from;
    size_t bytes;
};
// (Never destroyed: a program's static objects may give handles back at exit.)
std::mutex g_mu;                     // of all that follows
std::vector<std::unique_ptr<DevicePool>> &g_pools = *new std::vector<std::unique_ptr<DevicePool>>;
// What is live is counted here: the driver's own count (UsedMemCurrent) leaves out
// what cudaFree gives back.
std::unordered_map<void *, Allocation> &g_live = *new std::unordered_map<void *, Allocation>;

// The pool of the current device `dev`, made on first use.
int pool_of(int dev, DevicePool **out)
{
    if (dev < 0 || dev >= kMaxDevices) return MF_ERR_UNSUPPORTED;
    const MfContext ctx = mf_context();
    std::lock_guard<std::mutex> lock(g_mu);
    for (const auto &d : g_pools)
        if (d->dev == dev && d->ctx.object == ctx.object && d->ctx.id == ctx.id) {
            *out = d.get();
            return MF_SUCCESS;
        }
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
    g_pools.emplace_back(new DevicePool{dev, ctx, p, block, 0, 0});
    *out = g_pools.back().get();
    return MF_SUCCESS;
}

// The driver compares the release threshold with all the memory a pool holds,
// live allocations included.  With a fixed one, handles above it (three 128^3
// systems) had every freed array unmapped at the next synchronisation and mapped
// again for the next solve (first solve of a handle 4.9 -> 8.5 ms).
void follow(DevicePool *d)
{
    unsigned long long keep = d->live + kKeepBytes;
    if (cudaMemPoolSetAttribute(d->pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) cudaGetLastError();
}

constexpr size_t kFollowBytes = 4u << 20;    // allocations that move the threshold

void count_free(void *p)
{
    std::lock_guard<std::mutex> lock(g_mu);
    const auto it = g_live.find(p);
    if (it == g_live.end()) return;
    it->second.from->live -= it->second.bytes;
    g_live.erase(it);
}

// The driver's calls for a context and its id (null where the driver has none).
struct DriverCalls {
    int (*current)(void **) = nullptr;
    int (*id)(void *, unsigned long long *) = nullptr;
    DriverCalls()
    {
        cudaDriverEntryPointQueryResult q;
        void *f = nullptr, *g = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess && f &&
            cudaGetDriverEntryPointByVersion("cuCtxGetId", &g, 12000, cudaEnableDefault, &q) == cudaSuccess && g) {
            current = (int (*)(void **))f;
            id = (int (*)(void *, unsigned long long *))g;
        }
        cudaGetLastError();
    }
};

}  // namespace

// 14 ns a driver call.  Where there is no context yet, or a reset has ended it,
// cudaSetDevice makes one (no call that a stream capture forbids).
MfContext mf_context()
{
    static const DriverCalls driver;
    MfContext c = {nullptr, 0};
    if (!driver.id) return c;
    int dev = 0;
    if (driver.id(nullptr, &c.id) != 0 &&
        (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess || driver.id(nullptr, &c.id) != 0)) {
        cudaGetLastError();
        return {nullptr, 0};
    }
    if (driver.current(&c.object) != 0) return {nullptr, 0};
    return c;
}

bool mf_context_gone(const MfContext &c)
{
    const MfContext now = mf_context();
    return now.id != c.id && (now.object == c.object || now.id == 0);
}

int mf_pool_alloc(void **p, size_t bytes, cudaStream_t s)
{
    *p = nullptr;
    int dev = 0;
    MF_CUDA_TRY(cudaGetDevice(&dev));
    // On a captured stream the allocation would become a node of the graph: an address
    // without memory, kept by a handle whose call then fails at its synchronisation.
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaError_t cap = cudaStreamIsCapturing(s, &capture);
    if (cap == cudaSuccess && capture != cudaStreamCaptureStatusNone) cap = cudaErrorStreamCaptureUnsupported;
    if (cap != cudaSuccess) cudaGetLastError();
    MF_CUDA_TRY(cap);
    DevicePool *d = nullptr;
    const int rc = pool_of(dev, &d);
    if (rc != MF_SUCCESS) return rc;
    if (bytes == 0) bytes = 1;
    cudaError_t e = cudaMallocFromPoolAsync(p, bytes, d->pool, s);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        mf_device_wait();
        if (cudaMemPoolTrimTo(d->pool, 0) == cudaSuccess) e = cudaMallocFromPoolAsync(p, bytes, d->pool, s);
    }
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
    }
    MF_CUDA_TRY(e);
    std::lock_guard<std::mutex> lock(g_mu);
    g_live[*p] = {d, bytes};
    d->live += bytes;
    if (d->live > d->high) d->high = d->live;
    if (bytes >= kFollowBytes) follow(d);
    return MF_SUCCESS;
}

// An address is taken off the list before it goes back: from then on another
// thread may get it.
void mf_pool_free(void *p, cudaStream_t s)
{
    if (!p) return;
    count_free(p);
    if (cudaFreeAsync(p, s) != cudaSuccess) cudaGetLastError();
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
    for (int k = 0; k < count; k++) {
        if (!p[k]) continue;
        count_free(p[k]);
        if (cudaFree(p[k]) != cudaSuccess) cudaGetLastError();
    }
}

void mf_pool_settle(int dev)
{
    MfDeviceGuard guard(dev);
    DevicePool *d = nullptr;
    unsigned long long held = 0;
    if (pool_of(dev, &d) != MF_SUCCESS) return;
    std::lock_guard<std::mutex> lock(g_mu);
    follow(d);
    const unsigned long long keep =
        d->live > 0 ? d->live + kKeepBytes : d->high < kKeepBytes ? d->high : kKeepBytes;
    if (cudaMemPoolGetAttribute(d->pool, cudaMemPoolAttrReservedMemCurrent, &held) == cudaSuccess && held > keep)
        cudaMemPoolTrimTo(d->pool, (size_t)keep);
    if (d->live == 0) d->high = 0;
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
