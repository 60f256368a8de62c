#include "host_transfer.h"

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <map>
#include <mutex>
#include <new>
#include <stdexcept>
#include <string>
#include <system_error>
#include <thread>
#include <vector>

namespace vlrb {

namespace {

// One thread moves about 10 GB/s between pageable and pinned memory, the link
// about 50: four workers, two slots each so that one fills while the other
// travels.  Below kThreaded bytes a copy is over before a thread has started.
constexpr int kWorkers = 4, kSlotsPerWorker = 2, kSlots = kWorkers * kSlotsPerWorker;
constexpr size_t kChunk = size_t(1) << 20;
constexpr size_t kStaged = size_t(256) << 10, kThreaded = size_t(2) << 20;
// Rings and device blocks kept per CUDA context.  A ring takes milliseconds to make,
// so callers beyond the rings' number copy through the driver instead of
// making more (eight callers of 1,000 rays each: 2,470 us a call with rings of
// their own, 810 so).
constexpr int kRings = 2;
constexpr size_t kKeptBlocks = 8, kKeptBytes = size_t(256) << 20;

void ck(cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw std::runtime_error(std::string("host transfer ") + what + ": " + cudaGetErrorString(e));
}

} // namespace

// The CUDA context all handles and addresses belong to.  The id is never used
// again in a process: after cudaDeviceReset a device's primary context has the
// same handle and another id, and what was kept of the old one is gone with it.
struct CudaContext {
    CUcontext handle = nullptr;
    unsigned long long id = 0;
};

struct HostRing {
    CudaContext context;
    char* pinned = nullptr;
    cudaEvent_t done[kSlots] = {};
    bool used[kSlots] = {};

    ~HostRing() {
        for (cudaEvent_t e : done)
            if (e) cudaEventDestroy(e);
        if (pinned) cudaFreeHost(pinned);
    }
    char* slot(int s) const { return pinned + size_t(s) * kChunk; }
    void wait(int s) {
        if (used[s]) ck(cudaEventSynchronize(done[s]), "slot");
        used[s] = false;
    }
    void sent(int s) {
        ck(cudaEventRecord(done[s], nullptr), "slot");
        used[s] = true;
    }
};

namespace {

struct DeviceBlock {
    CudaContext context;
    void* p;
    size_t bytes;
};

// The driver's calls through the runtime (no link-time libcuda dependency).
struct Driver {
    CUresult (*getCurrent)(CUcontext*) = nullptr;
    CUresult (*setCurrent)(CUcontext) = nullptr;
    CUresult (*getId)(CUcontext, unsigned long long*) = nullptr;
};
template <class F>
void driverEntry(const char* name, F* fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    ck(cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q), name);
    if (!p) throw std::runtime_error(std::string("host transfer: no ") + name);
    *fn = reinterpret_cast<F>(p);
}
const Driver &driver() {
    static const Driver d = [] {
        Driver r;
        driverEntry("cuCtxGetCurrent", &r.getCurrent);
        driverEntry("cuCtxSetCurrent", &r.setCurrent);
        driverEntry("cuCtxGetId", &r.getId);
        return r;
    }();
    return d;
}

// The current context; false where there is none, or only the handle of one
// that is gone.
bool askContext(CudaContext* c) {
    return driver().getCurrent(&c->handle) == CUDA_SUCCESS && c->handle &&
           driver().getId(c->handle, &c->id) == CUDA_SUCCESS;
}

CudaContext currentContext() {
    CudaContext c;
    if (askContext(&c)) return c;
    ck(cudaFree(nullptr), "context");   // makes the device's primary context
    if (!askContext(&c)) throw std::runtime_error("host transfer: no CUDA context");
    return c;
}

// What is idle.  Never destroyed: the last context object may go after this
// library's static objects.
struct Kept {
    std::mutex mutex;
    std::vector<DeviceBlock> blocks;
    std::vector<HostRing*> rings;
    std::map<unsigned long long, int> ringsMade;   // per context, idle or borrowed
};
Kept &kept() {
    static Kept* const k = new Kept;
    return *k;
}

// Forgets what was kept of a context that is gone: its handle is `now`'s, its
// id is not.  (With the mutex held.)
void forgetGone(const CudaContext &now) {
    Kept &k = kept();
    auto gone = [&](const CudaContext &c) { return c.handle == now.handle && c.id != now.id; };
    k.blocks.erase(std::remove_if(k.blocks.begin(), k.blocks.end(), [&](const DeviceBlock &b) { return gone(b.context); }),
                   k.blocks.end());
    for (HostRing* &r : k.rings)
        if (gone(r->context)) {
            k.ringsMade.erase(r->context.id);
            r->pinned = nullptr;
            for (cudaEvent_t &e : r->done) e = nullptr;
            delete r;
            r = nullptr;
        }
    k.rings.erase(std::remove(k.rings.begin(), k.rings.end(), nullptr), k.rings.end());
}

// The smallest idle block of at least `bytes`.
bool takeBlock(const CudaContext &context, size_t bytes, DeviceBlock* out) {
    Kept &k = kept();
    std::lock_guard<std::mutex> lock(k.mutex);
    forgetGone(context);
    size_t best = k.blocks.size();
    for (size_t i = 0; i < k.blocks.size(); ++i)
        if (k.blocks[i].context.id == context.id && k.blocks[i].bytes >= bytes &&
            (best == k.blocks.size() || k.blocks[i].bytes < k.blocks[best].bytes))
            best = i;
    if (best == k.blocks.size()) return false;
    *out = k.blocks[best];
    k.blocks.erase(k.blocks.begin() + static_cast<std::ptrdiff_t>(best));
    return true;
}

// Keeps an idle block, in place of smaller ones where the limits ask for it.
void keepBlock(const DeviceBlock &block) {
    std::vector<void*> dropped;
    {
        Kept &k = kept();
        std::lock_guard<std::mutex> lock(k.mutex);
        size_t count = 0, bytes = 0, stayCount = 0, stayBytes = 0;
        for (const DeviceBlock &b : k.blocks)
            if (b.context.id == block.context.id) {
                ++count;
                bytes += b.bytes;
                if (b.bytes >= block.bytes) { ++stayCount; stayBytes += b.bytes; }
            }
        const bool fits = stayCount + 1 <= kKeptBlocks && stayBytes + block.bytes <= kKeptBytes;
        while (fits && (count + 1 > kKeptBlocks || bytes + block.bytes > kKeptBytes)) {
            auto least = k.blocks.end();
            for (auto i = k.blocks.begin(); i != k.blocks.end(); ++i)
                if (i->context.id == block.context.id && i->bytes < block.bytes &&
                    (least == k.blocks.end() || i->bytes < least->bytes))
                    least = i;
            --count;
            bytes -= least->bytes;
            dropped.push_back(least->p);
            k.blocks.erase(least);
        }
        if (fits) k.blocks.push_back(block);
        else dropped.push_back(block.p);
    }
    for (void* p : dropped) cudaFree(p);
}

// An idle ring, a new one, or null: the caller then copies through the driver.
HostRing* takeRing(const CudaContext &context) {
    Kept &k = kept();
    {
        std::lock_guard<std::mutex> lock(k.mutex);
        for (size_t i = 0; i < k.rings.size(); ++i)
            if (k.rings[i]->context.id == context.id) {
                HostRing* r = k.rings[i];
                k.rings.erase(k.rings.begin() + static_cast<std::ptrdiff_t>(i));
                return r;
            }
        if (k.ringsMade[context.id] >= kRings) return nullptr;
        ++k.ringsMade[context.id];
    }
    HostRing* r = new HostRing;
    r->context = context;
    bool ok = cudaMallocHost(reinterpret_cast<void**>(&r->pinned), kSlots * kChunk) == cudaSuccess;
    for (int i = 0; ok && i < kSlots; ++i)
        ok = cudaEventCreateWithFlags(&r->done[i], cudaEventDisableTiming) == cudaSuccess;
    if (ok) return r;
    cudaGetLastError();
    delete r;
    std::lock_guard<std::mutex> lock(k.mutex);
    --k.ringsMade[context.id];
    return nullptr;
}

void returnRing(HostRing* r, bool idle) {
    Kept &k = kept();
    std::lock_guard<std::mutex> lock(k.mutex);
    if (idle) { k.rings.push_back(r); return; }
    --k.ringsMade[r->context.id];
    delete r;
}

// Whether the CPU may stage the array: pinned memory moves by itself at the
// link's rate, and device memory given as an array is the driver's to judge.
bool pageable(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) == cudaSuccess) return a.type == cudaMemoryTypeUnregistered;
    cudaGetLastError();
    return false;
}

// Runs work(worker) in this thread and, for a large copy, in kWorkers - 1
// others; the first exception is rethrown when all have ended.
template <class F>
void runWorkers(const CudaContext &context, size_t bytes, F work) {
    int n = bytes < kThreaded ? 1 : std::min<int>(kWorkers, static_cast<int>((bytes + kChunk - 1) / kChunk));
    n = std::min<int>(n, std::max<int>(1, static_cast<int>(std::thread::hardware_concurrency()) / 2));
    std::exception_ptr failed[kWorkers];
    auto guarded = [&](int worker) {
        try {
            if (worker > 0 && driver().setCurrent(context.handle) != CUDA_SUCCESS)
                throw std::runtime_error("host transfer: worker without the caller's context");
            work(worker);
        }
        catch (...) {
            failed[worker] = std::current_exception();
        }
    };
    std::thread threads[kWorkers - 1];
    int started = 0;
    try {
        for (; started + 1 < n; ++started) threads[started] = std::thread(guarded, started + 1);
    }
    catch (const std::system_error &) {
        // no more threads: those that run share the work
    }
    guarded(0);
    for (int i = 0; i < started; ++i) threads[i].join();
    for (const std::exception_ptr &e : failed)
        if (e) std::rethrow_exception(e);
}

} // namespace

void releaseHostTransfers() noexcept {
    std::vector<void*> blocks;
    std::vector<HostRing*> rings;
    try {
        Kept &k = kept();
        {
            std::lock_guard<std::mutex> lock(k.mutex);
            if (k.blocks.empty() && k.rings.empty()) return;
        }
        CudaContext now;
        if (!askContext(&now)) return;
        std::lock_guard<std::mutex> lock(k.mutex);
        forgetGone(now);
        blocks.reserve(k.blocks.size());
        rings.reserve(k.rings.size());
        for (size_t i = k.blocks.size(); i-- > 0;)
            if (k.blocks[i].context.id == now.id) {
                blocks.push_back(k.blocks[i].p);
                k.blocks.erase(k.blocks.begin() + static_cast<std::ptrdiff_t>(i));
            }
        for (size_t i = k.rings.size(); i-- > 0;)
            if (k.rings[i]->context.id == now.id) {
                rings.push_back(k.rings[i]);
                k.rings.erase(k.rings.begin() + static_cast<std::ptrdiff_t>(i));
                --k.ringsMade[now.id];
            }
    }
    catch (...) {
        return;   // no driver left to ask (the process ends), or no memory: nothing is released
    }
    for (void* p : blocks) cudaFree(p);
    for (HostRing* r : rings) delete r;
}

cudaError_t deviceMalloc(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    releaseHostTransfers();
    e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

HostTransfer::HostTransfer(size_t deviceBytes) {
    const CudaContext context = currentContext();
    contextHandle = context.handle;
    contextId = context.id;
    DeviceBlock block{ context, nullptr, deviceBytes };
    if (!takeBlock(context, deviceBytes, &block)) {
        ck(deviceMalloc(&block.p, deviceBytes), "workspace");
    }
    dev = block.p;
    devBytes = block.bytes;
}

HostTransfer::~HostTransfer() {
    // nothing of this call may still use what another takes
    const bool idle = cudaStreamSynchronize(nullptr) == cudaSuccess;
    try {
        if (ring) returnRing(ring, idle);
        if (idle) keepBlock(DeviceBlock{ { contextHandle, contextId }, dev, devBytes });
        else cudaFree(dev);
    }
    catch (const std::bad_alloc &) {
        // no host memory to note what is kept: it is not
    }
}

void* HostTransfer::device() const { return dev; }

bool HostTransfer::staged(const void* array, size_t bytes) {
    if (bytes < kStaged || !pageable(array)) return false;
    if (!ring && !ringAsked) ring = takeRing({ contextHandle, contextId });
    ringAsked = true;
    return ring != nullptr;
}

void HostTransfer::upload(void* dst, const void* src, size_t bytes) {
    if (!staged(src, bytes)) {
        if (bytes) ck(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, nullptr), "upload");
        return;
    }
    HostRing* const w = ring;
    std::atomic<size_t> next{ 0 };
    runWorkers(w->context, bytes, [&](int worker) {
        for (int turn = 0;; ++turn) {
            const size_t at = next.fetch_add(1) * kChunk;
            if (at >= bytes) return;
            const size_t len = std::min(kChunk, bytes - at);
            const int s = worker * kSlotsPerWorker + turn % kSlotsPerWorker;
            w->wait(s);
            std::memcpy(w->slot(s), static_cast<const char*>(src) + at, len);
            ck(cudaMemcpyAsync(static_cast<char*>(dst) + at, w->slot(s), len, cudaMemcpyHostToDevice, nullptr), "upload");
            w->sent(s);
        }
    });
}

void HostTransfer::download(void* dst, const void* src, size_t bytes) {
    if (!staged(dst, bytes)) {
        if (bytes) ck(cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToHost), "download");
        return;
    }
    HostRing* const w = ring;
    std::atomic<size_t> next{ 0 };
    runWorkers(w->context, bytes, [&](int worker) {
        size_t pendingAt = 0, pendingLen = 0;
        int pending = -1;
        auto drain = [&] {
            if (pending < 0) return;
            w->wait(pending);
            std::memcpy(static_cast<char*>(dst) + pendingAt, w->slot(pending), pendingLen);
            pending = -1;
        };
        for (int turn = 0;; ++turn) {
            const size_t at = next.fetch_add(1) * kChunk;
            if (at >= bytes) break;
            const size_t len = std::min(kChunk, bytes - at);
            const int s = worker * kSlotsPerWorker + turn % kSlotsPerWorker;
            w->wait(s);
            ck(cudaMemcpyAsync(w->slot(s), static_cast<const char*>(src) + at, len, cudaMemcpyDeviceToHost, nullptr),
               "download");
            w->sent(s);
            drain();   // the chunk before, while this one travels
            pending = s;
            pendingAt = at;
            pendingLen = len;
        }
        drain();
    });
}

} // namespace vlrb
