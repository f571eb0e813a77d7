// Transfers between ordinary (pageable) host memory and the device.
//
// The reference wraps every host array in an OpenCL buffer per call
// (core/src/ocl/ocl_buffer.cpp:27-42) and reads the outputs back before
// returning (core/src/ocl/ocl_kernel.cpp:59-111); a drop-in caller therefore
// passes ordinary malloc'd memory.  A DMA engine can only read page-locked
// memory, so such a copy goes through pinned memory either way.  Large copies
// use two pinned bounce buffers that each handle owns: while the DMA engine
// moves one buffer, host threads of a process-wide pool copy the next chunk
// into (or out of) the other, so the host-side copies and the PCIe transfers
// overlap.  Operands below the size of such a pipeline take 1 MiB chunks of
// a small process-wide pool of pinned memory instead, copied by the same
// threads (the driver copies them on one thread: 11 to 14 GB/s; a product of
// 1024 x 768 x 512 on host arrays takes 287 us so, 510 through the driver).
#include <algorithm>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "copy_pool.h"
#include "internal.h"

namespace iclb {
namespace {

constexpr size_t kBounceBytes = (size_t)32 << 20;   // one bounce buffer

// The process-wide pool of copy threads, started on first use.
CopyPool& copy_pool()
{
    static CopyPool pool(std::min(8u, std::max(2u, std::thread::hardware_concurrency()) / 2),
                         [](void* dst, const void* src, size_t bytes) { std::memcpy(dst, src, bytes); });
    return pool;
}

// Process-wide pool of pinned chunks for small copies: at most kMaxChunks, made
// as they are needed, given back to the system when the last handle goes.  A
// call holds a chunk until its DMA is over; with none left the caller copies
// through the driver.
class PinnedPool {
public:
    static PinnedPool& get()
    {
        static PinnedPool* pool = new PinnedPool();  // never destroyed: handles may outlive static objects
        return *pool;
    }
    void retain()
    {
        std::lock_guard<std::mutex> lock(mu_);
        ++handles_;
    }
    void release()
    {
        std::lock_guard<std::mutex> lock(mu_);
        if (--handles_ > 0) return;
        for (void* c : free_)
            if (cudaFreeHost(c) != cudaSuccess) cudaGetLastError();
        made_ -= (int)free_.size();
        free_.clear();
    }
    void* take()
    {
        std::lock_guard<std::mutex> lock(mu_);
        if (!free_.empty()) {
            void* c = free_.back();
            free_.pop_back();
            return c;
        }
        if (made_ >= kMaxChunks) return nullptr;
        void* c = nullptr;
        if (cudaHostAlloc(&c, kPinnedChunk, cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        ++made_;
        return c;
    }
    void give(void* c)
    {
        std::lock_guard<std::mutex> lock(mu_);
        free_.push_back(c);
    }

private:
    static constexpr int kMaxChunks = 16;
    std::mutex mu_;
    std::vector<void*> free_;
    int made_ = 0, handles_ = 0;
};

cudaError_t ensure_bounce(iclblasHandle_t h)
{
    for (int b = 0; b < 2; ++b) {
        cudaError_t e;
        if (!h->bounce[b] && (e = cudaHostAlloc(&h->bounce[b], kBounceBytes, cudaHostAllocDefault)) != cudaSuccess)
            return e;
        if (!h->bounce_ev[b] && (e = cudaEventCreateWithFlags(&h->bounce_ev[b], cudaEventDisableTiming)) != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

// Waits until the copy that last used bounce buffer b has finished with it.
cudaError_t bounce_free(iclblasHandle_t h, int b)
{
    if (!h->bounce_busy[b]) return cudaSuccess;
    h->bounce_busy[b] = false;
    return cudaEventSynchronize(h->bounce_ev[b]);
}

}  // namespace

void pinned_retain() { PinnedPool::get().retain(); }
void pinned_release() { PinnedPool::get().release(); }
void* pinned_take() { return PinnedPool::get().take(); }
void pinned_give(void* chunk) { PinnedPool::get().give(chunk); }

void host_copy(void* dst, const void* src, size_t bytes) { copy_pool().copy(dst, src, bytes); }

cudaError_t copy_pageable_h2d(iclblasHandle_t h, void* dst, const void* src, size_t bytes)
{
    cudaError_t e = ensure_bounce(h);
    if (e != cudaSuccess) return e;
    size_t off = 0;
    for (int i = 0; off < bytes; ++i) {
        const int b = i & 1;
        const size_t len = std::min(kBounceBytes, bytes - off);
        if ((e = bounce_free(h, b)) != cudaSuccess) return e;
        host_copy(h->bounce[b], (const char*)src + off, len);
        if ((e = cudaMemcpyAsync((char*)dst + off, h->bounce[b], len, cudaMemcpyHostToDevice, h->stream)) !=
            cudaSuccess)
            return e;
        if ((e = cudaEventRecord(h->bounce_ev[b], h->stream)) != cudaSuccess) return e;
        h->bounce_busy[b] = true;
        off += len;
    }
    return cudaSuccess;
}

cudaError_t copy_pageable_d2h(iclblasHandle_t h, void* dst, const void* src, size_t bytes)
{
    cudaError_t e = ensure_bounce(h);
    if (e != cudaSuccess) return e;
    const int nchunks = (int)((bytes + kBounceBytes - 1) / kBounceBytes);
    auto issue = [&](int i) -> cudaError_t {
        const int b = i & 1;
        const size_t off = (size_t)i * kBounceBytes, len = std::min(kBounceBytes, bytes - off);
        cudaError_t r = bounce_free(h, b);
        if (r != cudaSuccess) return r;
        if ((r = cudaMemcpyAsync(h->bounce[b], (const char*)src + off, len, cudaMemcpyDeviceToHost, h->stream)) !=
            cudaSuccess)
            return r;
        if ((r = cudaEventRecord(h->bounce_ev[b], h->stream)) != cudaSuccess) return r;
        h->bounce_busy[b] = true;
        return cudaSuccess;
    };
    if (nchunks > 0 && (e = issue(0)) != cudaSuccess) return e;
    for (int i = 0; i < nchunks; ++i) {
        // the DMA of chunk i + 1 runs while chunk i is copied out
        if (i + 1 < nchunks && (e = issue(i + 1)) != cudaSuccess) return e;
        const int b = i & 1;
        if ((e = cudaEventSynchronize(h->bounce_ev[b])) != cudaSuccess) return e;
        const size_t off = (size_t)i * kBounceBytes, len = std::min(kBounceBytes, bytes - off);
        host_copy((char*)dst + off, h->bounce[b], len);
        h->bounce_busy[b] = false;
    }
    return cudaSuccess;
}

cudaError_t free_bounce(iclblasHandle_t h)
{
    cudaError_t r = cudaSuccess;
    for (int b = 0; b < 2; ++b) {
        if (h->bounce_ev[b]) {
            cudaEventSynchronize(h->bounce_ev[b]);
            cudaEventDestroy(h->bounce_ev[b]);
            h->bounce_ev[b] = nullptr;
        }
        if (h->bounce[b]) {
            cudaError_t e = cudaFreeHost(h->bounce[b]);
            if (r == cudaSuccess) r = e;
            h->bounce[b] = nullptr;
        }
        h->bounce_busy[b] = false;
    }
    return r;
}

}  // namespace iclb
