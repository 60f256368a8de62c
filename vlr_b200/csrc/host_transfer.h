// Device workspace and host copies of the entry points that take host arrays.
//
// Those calls were bound by what surrounds their kernels: device allocations
// and frees made and undone every call, and copies between pageable memory and
// the device, which the driver stages through one thread.  A HostTransfer
// borrows for one call a device block kept from earlier calls and, once it has
// a large pageable array to move, a ring of pinned slots that several threads
// fill or drain while the copy engine works on the others.  With the same
// kernels, numpy callers and pageable arrays: one million rays against 20,022
// triangles (32 MB in, 16 MB out, the hierarchy built on the way) 8.4 -> 5.4 ms;
// the hierarchy of 150,001 triangles 4.4 -> 2.7 ms; 65,536 queries and gradients
// of the guiding network 4.0 -> 2.5 ms.  Pinned arrays go as they are: the same
// rays, the call alone, 4.1 ms from pageable arrays and 2.9 from pinned ones.
//
// Blocks and rings belong to a CUDA context, and are forgotten when it is gone
// (cudaDeviceReset); a call has its own, so calls from several threads run side by
// side.  What is kept is bounded: two rings (calls that find
// both in use copy through the driver), and at most eight blocks of 256 MB in
// all; a larger block is freed when its call ends.  It is given back when an
// allocation of the library fails, and with the last context object.
// All work is on the legacy default stream, which orders it after other
// blocking streams' work as cudaMemcpy does.
#pragma once

#include <cstddef>

#include <cuda_runtime.h>

struct CUctx_st;

namespace vlrb {

struct HostRing;

class HostTransfer {
public:
    // Throws std::runtime_error when the device has no memory left.
    explicit HostTransfer(size_t deviceBytes);
    ~HostTransfer();
    HostTransfer(const HostTransfer &) = delete;
    HostTransfer &operator=(const HostTransfer &) = delete;

    void* device() const;
    // Enqueues the copy.  `src` may be read until the next download or the end of
    // this object, and must stay as it is until then.  Pageable arrays are staged;
    // any other memory goes to the driver as it is.
    void upload(void* dst, const void* src, size_t bytes);
    // Returns once `dst` holds the bytes the stream's earlier work left at `src`.
    void download(void* dst, const void* src, size_t bytes);

private:
    bool staged(const void* array, size_t bytes);

    CUctx_st* contextHandle = nullptr;
    unsigned long long contextId = 0;
    void* dev = nullptr;
    size_t devBytes = 0;
    HostRing* ring = nullptr;
    bool ringAsked = false;
};

// Frees the idle blocks and rings kept for the current CUDA context (called from
// destructors too, at the process's end among them).
void releaseHostTransfers() noexcept;

// cudaMalloc; when there is no memory left, once more without what is kept.
cudaError_t deviceMalloc(void** p, size_t bytes);

} // namespace vlrb
