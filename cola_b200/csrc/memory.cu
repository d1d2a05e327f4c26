// Device memory of the library: one stream-ordered pool per device that keeps
// up to kKeep bytes mapped after they are freed.  Mapping and unmapping cost
// about 7 ms a gigabyte each with the default pool (which unmaps at every
// synchronisation) and 0.3 to 0.6 ms per cudaMalloc or cudaFree of 16 to 480 MB,
// most of the wall time of building a graph (1 M rows, 14 M entries, and one
// SpMM: 4.8 ms and up to 29 on a busy host, 1.7 with the pool).  The kept bytes
// are given back by cola_trim_memory and before the library reports that the
// device is full; the driver gives back what exceeds kKeep at each
// synchronisation.  Pools are safe with several threads and streams: memory freed
// on one stream is handed to another only in order.
#include <mutex>

#include <cuda_runtime.h>

#include "common.h"
#include "graph.h"

namespace cola {

constexpr unsigned long long kKeep = 1ull << 30;
constexpr int kMaxDevices = 64;

struct DevicePool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;  // allocations that outlive a call are made on it
    void *anchor = nullptr;         // keeps the driver's chunk of small blocks, see wait_device
    bool tried = false;
    unsigned long long context = 0;  // the context they belong to
};

static std::mutex g_pool_mu;
static DevicePool g_pools[kMaxDevices];

// The current device's pool; its members are NULL where it cannot be had.  One
// that went with its context (cudaDeviceReset) is not used again.
static DevicePool device_pool_entry()
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return DevicePool();
    unsigned long long context = current_context_id();
    if (context == 0) {
        cudaFree(nullptr);  // makes the device's context
        context = current_context_id();
    }
    std::lock_guard<std::mutex> lk(g_pool_mu);
    DevicePool &p = g_pools[dev];
    if (!p.tried || p.context != context) {
        p = DevicePool();
        p.tried = true;
        p.context = context;
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        unsigned long long keep = kKeep;
        if (cudaMemPoolCreate(&p.pool, &props) != cudaSuccess ||
            cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
            cudaStreamCreateWithFlags(&p.stream, cudaStreamNonBlocking) != cudaSuccess) {
            cudaGetLastError();
            if (p.pool)
                cudaMemPoolDestroy(p.pool);
            p.pool = nullptr;
            p.stream = nullptr;
        }
        if (cudaMalloc(&p.anchor, 256) != cudaSuccess)
            cudaGetLastError();
    }
    return p;
}

// Lets the calling thread allocate and free while a stream is being captured
// (in the default mode such a call is refused and ends the capture).
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Waits for the work on every stream of the current device.
// cudaDeviceSynchronize is refused while any stream of the device is being
// captured, and ends that capture, whichever thread calls it and whatever the
// capture's mode; cudaFree of a block from cudaMalloc waits for all streams too
// (a 20 ms kernel on a non-blocking stream: 20 ms) and leaves captures alone.
// 3.7 us on an idle device, with the block's chunk kept mapped by `anchor`.
static bool wait_device()
{
    void *p = nullptr;
    const cudaError_t e = cudaMalloc(&p, 256) == cudaSuccess ? cudaFree(p) : cudaDeviceSynchronize();
    cudaGetLastError();
    return e == cudaSuccess;
}

// Unmaps what the pool keeps and nobody uses.
static void trim(const DevicePool &p)
{
    const RelaxedCapture relaxed;
    if (p.pool && wait_device())
        cudaMemPoolTrimTo(p.pool, 0);
    cudaGetLastError();
}

// Requests past kPooled go to cudaMalloc and cudaFree: about 1 ms each at 700 MB,
// where the pool, which keeps no more than kKeep, would map and unmap for 10.
constexpr size_t kPooled = kKeep / 2;

cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t st)
{
    const DevicePool dp = device_pool_entry();
    if (bytes > kPooled) {
        cudaError_t e = cudaMalloc(p, bytes);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            trim(dp);
            e = cudaMalloc(p, bytes);
        }
        return e;
    }
    if (!dp.pool)
        return cudaMallocAsync(p, bytes, st);
    cudaError_t e = cudaMallocFromPoolAsync(p, bytes, dp.pool, st);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        trim(dp);
        e = cudaMallocFromPoolAsync(p, bytes, dp.pool, st);
    }
    return e;
}

void scratch_free(void *p, size_t bytes, cudaStream_t st)
{
    if (bytes > kPooled) {
        cudaStreamSynchronize(st);
        cudaFree(p);
    } else {
        cudaFreeAsync(p, st);
    }
}

cudaError_t device_alloc(void **p, size_t bytes)
{
    const RelaxedCapture relaxed;
    const DevicePool dp = device_pool_entry();
    if (dp.pool && bytes <= kPooled) {
        if (cudaMallocFromPoolAsync(p, bytes, dp.pool, dp.stream) == cudaSuccess) {
            const cudaError_t e = cudaStreamSynchronize(dp.stream);  // usable on every stream from here on
            if (e != cudaSuccess)
                cudaFreeAsync(*p, dp.stream);
            return e;
        }
        cudaGetLastError();
    }
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation && dp.pool) {
        cudaGetLastError();
        trim(dp);
        e = cudaMalloc(p, bytes);
    }
    return e;
}

void device_free(void *p)
{
    if (!p)
        return;
    const RelaxedCapture relaxed;
    // cudaFree waits for the device itself only for memory from cudaMalloc
    if (wait_device())
        cudaFree(p);
    cudaGetLastError();
}

}  // namespace cola

extern "C" cola_status cola_trim_memory(void)
{
    cola::trim(cola::device_pool_entry());
    return COLA_SUCCESS;
}
