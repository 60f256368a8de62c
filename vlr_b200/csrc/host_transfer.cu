#include "host_transfer.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
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
constexpr size_t kKept = 2, kKeptBytes = size_t(256) << 20;

void ck(cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw std::runtime_error(std::string("host transfer ") + what + ": " + cudaGetErrorString(e));
}

} // namespace

struct HostWorkspace {
    int device = 0;
    void* dev = nullptr;
    size_t devBytes = 0;
    char* pinned = nullptr;
    cudaEvent_t done[kSlots] = {};
    bool used[kSlots] = {};

    ~HostWorkspace() {
        for (cudaEvent_t e : done)
            if (e) cudaEventDestroy(e);
        if (pinned) cudaFreeHost(pinned);
        if (dev) cudaFree(dev);
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

std::mutex g_mutex;
std::vector<HostWorkspace*> g_free;   // kept to the end of the process

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
void runWorkers(int device, size_t bytes, F work) {
    int n = bytes < kThreaded ? 1 : std::min<int>(kWorkers, static_cast<int>((bytes + kChunk - 1) / kChunk));
    n = std::min<int>(n, std::max<int>(1, static_cast<int>(std::thread::hardware_concurrency()) / 2));
    std::exception_ptr failed[kWorkers];
    auto guarded = [&](int worker) {
        try {
            if (worker > 0) ck(cudaSetDevice(device), "device");
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

HostTransfer::HostTransfer(size_t deviceBytes) : w(nullptr) {
    int device = 0;
    ck(cudaGetDevice(&device), "device");
    {
        // the smallest kept workspace that is large enough, else the largest
        std::lock_guard<std::mutex> lock(g_mutex);
        size_t best = g_free.size();
        for (size_t i = 0; i < g_free.size(); ++i) {
            if (g_free[i]->device != device) continue;
            if (best == g_free.size()) { best = i; continue; }
            const size_t a = g_free[i]->devBytes, b = g_free[best]->devBytes;
            if (a >= deviceBytes ? (b < deviceBytes || a < b) : (b < deviceBytes && a > b)) best = i;
        }
        if (best < g_free.size()) {
            w = g_free[best];
            g_free.erase(g_free.begin() + static_cast<std::ptrdiff_t>(best));
        }
    }
    if (!w) {
        w = new HostWorkspace;
        w->device = device;
    }
    try {
        if (!w->pinned) {
            ck(cudaMallocHost(reinterpret_cast<void**>(&w->pinned), kSlots * kChunk), "pinned memory");
            for (cudaEvent_t &e : w->done) ck(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "event");
        }
        if (w->devBytes < deviceBytes) {
            if (w->dev) cudaFree(w->dev);
            w->dev = nullptr;
            w->devBytes = 0;
            ck(cudaMalloc(&w->dev, deviceBytes), "workspace");
            w->devBytes = deviceBytes;
        }
    }
    catch (...) {
        delete w;
        cudaGetLastError();
        throw;
    }
}

HostTransfer::~HostTransfer() {
    // nothing of this call may still use the buffers when another takes them
    const bool idle = cudaStreamSynchronize(nullptr) == cudaSuccess;
    if (idle && w->devBytes <= kKeptBytes) {
        std::lock_guard<std::mutex> lock(g_mutex);
        size_t kept = 0;
        for (const HostWorkspace* f : g_free) kept += f->device == w->device;
        if (kept < kKept) {
            g_free.push_back(w);
            return;
        }
    }
    delete w;
}

void* HostTransfer::device() const { return w->dev; }

void HostTransfer::upload(void* dst, const void* src, size_t bytes) {
    if (bytes < kStaged || !pageable(src)) {
        if (bytes) ck(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, nullptr), "upload");
        return;
    }
    std::atomic<size_t> next{ 0 };
    runWorkers(w->device, bytes, [&](int worker) {
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
    if (bytes < kStaged || !pageable(dst)) {
        if (bytes) ck(cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToHost), "download");
        return;
    }
    std::atomic<size_t> next{ 0 };
    runWorkers(w->device, bytes, [&](int worker) {
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
