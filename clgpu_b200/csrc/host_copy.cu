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
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "internal.h"

namespace iclb {
namespace {

constexpr size_t kBounceBytes = (size_t)32 << 20;   // one bounce buffer
constexpr size_t kSliceBytes = (size_t)128 << 10;   // least host-copy work per thread and copy
constexpr int kSpinUs = 50;                         // a worker looks for the next copy this long before it sleeps

inline void cpu_pause()
{
#if defined(__x86_64__)
    __builtin_ia32_pause();
#else
    std::this_thread::yield();
#endif
}

// Process-wide pool of host threads for memcpy calls (started on first use).
// One copy at a time is shared out: the slices of it that are still to be
// done are handed out by an atomic counter, to the workers that come and to
// the caller itself, so the caller never waits for a thread that has yet to
// wake up, and no lock is taken on the way (with a locked queue, eight
// workers waking up for a 1 MiB copy cost more than the copy).  A caller that
// finds the pool taken copies on its own thread.  Workers spin for kSpinUs
// after a copy: the next chunk of the same call finds them awake.
class CopyPool {
public:
    static CopyPool& get()
    {
        static CopyPool pool;
        return pool;
    }

    void copy(void* dst, const void* src, size_t bytes)
    {
        const size_t n = std::min<size_t>(workers_.size() + 1, (bytes + kSliceBytes - 1) / kSliceBytes);
        std::unique_lock<std::mutex> mine(owner_, std::defer_lock);
        if (n <= 1 || !mine.try_lock()) {
            std::memcpy(dst, src, bytes);
            return;
        }
        dst_ = (char*)dst;
        src_ = (const char*)src;
        bytes_ = bytes;
        per_ = ((bytes + n - 1) / n + 63) & ~(size_t)63;
        slices_ = (int)((bytes + per_ - 1) / per_);
        next_.store(0);
        done_.store(0);
        open_.store(true);      // workers may enter
        copies_.fetch_add(1);   // and know there is something new
        if (sleeping_.load() > 0) {
            std::lock_guard<std::mutex> lock(mu_);
            cv_.notify_all();
        }
        work();
        while (done_.load() < slices_) cpu_pause();
        // no worker may look at this copy once the next one is set up
        open_.store(false);
        while (inside_.load() > 0) cpu_pause();
    }

    ~CopyPool()
    {
        {
            std::lock_guard<std::mutex> lock(mu_);
            stop_.store(true);
        }
        cv_.notify_all();
        for (auto& t : workers_) t.join();
    }

private:
    CopyPool()
    {
        const unsigned hw = std::max(2u, std::thread::hardware_concurrency());
        const unsigned n = std::min(8u, hw / 2);
        for (unsigned i = 0; i < n; ++i) workers_.emplace_back([this] { run(); });
    }

    void work()
    {
        for (int i = next_.fetch_add(1); i < slices_; i = next_.fetch_add(1)) {
            const size_t off = (size_t)i * per_;
            std::memcpy(dst_ + off, src_ + off, std::min(per_, bytes_ - off));
            done_.fetch_add(1);
        }
    }

    void run()
    {
        unsigned seen = 0;
        for (;;) {
            const auto t0 = std::chrono::steady_clock::now();
            while (copies_.load() == seen && !stop_.load() &&
                   std::chrono::steady_clock::now() - t0 < std::chrono::microseconds(kSpinUs))
                cpu_pause();
            if (copies_.load() == seen) {
                std::unique_lock<std::mutex> lock(mu_);
                sleeping_.fetch_add(1);
                cv_.wait(lock, [&] { return stop_.load() || copies_.load() != seen; });
                sleeping_.fetch_sub(1);
            }
            if (stop_.load()) return;
            seen = copies_.load();
            // the caller closes the copy and then waits for inside_ == 0: a
            // worker that still finds it open is waited for
            inside_.fetch_add(1);
            if (open_.load()) work();
            inside_.fetch_sub(1);
        }
    }

    std::mutex owner_;  // held by the caller whose copy is shared out
    char* dst_ = nullptr;
    const char* src_ = nullptr;
    size_t bytes_ = 0, per_ = 0;
    int slices_ = 0;
    std::atomic<int> next_{0}, done_{0}, inside_{0}, sleeping_{0};
    std::atomic<unsigned> copies_{0};
    std::atomic<bool> open_{false}, stop_{false};
    std::mutex mu_;
    std::condition_variable cv_;
    std::vector<std::thread> workers_;
};

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

void host_copy(void* dst, const void* src, size_t bytes) { CopyPool::get().copy(dst, src, bytes); }

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
