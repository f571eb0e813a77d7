// Host threads that share out memcpy calls.
//
// Kept free of CUDA headers so that the sharing can be compiled and checked on
// a machine without a GPU.  Each copy under way has a place of its own: its
// slices are handed out by an atomic counter, to the workers that come and to
// the caller itself, so a caller never waits for a thread that has yet to wake
// up, and no lock is taken on the way (with a locked queue, eight workers
// waking up for a 1 MiB copy cost more than the copy).  Workers go from copy to
// copy a slice at a time, so several callers share them evenly; only a caller
// that finds all places taken copies on its own thread.  Workers spin for
// kSpinUs after a copy: the next chunk of the same call finds them awake.
#pragma once

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstddef>
#include <mutex>
#include <thread>
#include <vector>

namespace iclb {

class CopyPool {
public:
    using CopyFn = void (*)(void* dst, const void* src, size_t bytes);

    CopyPool(unsigned workers, CopyFn fn) : fn_(fn)
    {
        for (unsigned i = 0; i < workers; ++i) workers_.emplace_back([this, i] { run(i); });
    }
    CopyPool(const CopyPool&) = delete;
    CopyPool& operator=(const CopyPool&) = delete;
    ~CopyPool()
    {
        {
            std::lock_guard<std::mutex> lock(mu_);
            stop_.store(true);
        }
        cv_.notify_all();
        for (auto& t : workers_) t.join();
    }

    void copy(void* dst, const void* src, size_t bytes)
    {
        const size_t n = std::min<size_t>(workers_.size() + 1, (bytes + kSliceBytes - 1) / kSliceBytes);
        Place* p = n > 1 ? take() : nullptr;
        if (!p) {
            fn_(dst, src, bytes);
            return;
        }
        p->dst = (char*)dst;
        p->src = (const char*)src;
        p->bytes = bytes;
        p->per = ((bytes + n - 1) / n + 63) & ~(size_t)63;
        p->slices = (int)((bytes + p->per - 1) / p->per);
        p->next.store(0);
        p->done.store(0);
        p->open.store(true);    // workers may enter
        copies_.fetch_add(1);   // and know there is something new
        if (sleeping_.load() > 0) {
            std::lock_guard<std::mutex> lock(mu_);
            cv_.notify_all();
        }
        while (slice(*p)) {}
        while (p->done.load() < p->slices) pause();
        // no worker may look at this copy once the next one is set up
        p->open.store(false);
        while (p->inside.load() > 0) pause();
        p->owner.unlock();
    }

private:
    static constexpr int kPlaces = 8;                           // copies that share the workers
    static constexpr size_t kSliceBytes = (size_t)128 << 10;    // least work per thread and copy
    static constexpr int kSpinUs = 50;                          // a worker looks for the next copy this long

    struct Place {
        std::mutex owner;  // held by the caller whose copy it is
        char* dst = nullptr;
        const char* src = nullptr;
        size_t bytes = 0, per = 0;
        int slices = 0;
        std::atomic<int> next{0}, done{0}, inside{0};
        std::atomic<bool> open{false};
    };

    static void pause()
    {
#if defined(__x86_64__)
        __builtin_ia32_pause();
#else
        std::this_thread::yield();
#endif
    }

    Place* take()
    {
        for (Place& p : places_)
            if (p.owner.try_lock()) return &p;
        return nullptr;
    }

    // copies one slice of p that is still to be done
    bool slice(Place& p)
    {
        const int i = p.next.fetch_add(1);
        if (i >= p.slices) return false;
        const size_t off = (size_t)i * p.per;
        fn_(p.dst + off, p.src + off, std::min(p.per, p.bytes - off));
        p.done.fetch_add(1);
        return true;
    }

    void run(unsigned at)
    {
        unsigned seen = 0;
        for (;;) {
            const auto t0 = std::chrono::steady_clock::now();
            while (copies_.load() == seen && !stop_.load() &&
                   std::chrono::steady_clock::now() - t0 < std::chrono::microseconds(kSpinUs))
                pause();
            if (copies_.load() == seen) {
                std::unique_lock<std::mutex> lock(mu_);
                sleeping_.fetch_add(1);
                cv_.wait(lock, [&] { return stop_.load() || copies_.load() != seen; });
                sleeping_.fetch_sub(1);
            }
            if (stop_.load()) return;
            seen = copies_.load();
            // a slice of each open copy in turn, until a round finds none
            for (int none = 0; none < kPlaces; ++at) {
                Place& p = places_[at % kPlaces];
                bool did = false;
                if (p.open.load()) {
                    // the caller closes the copy and then waits for inside == 0:
                    // a worker that still finds it open is waited for
                    p.inside.fetch_add(1);
                    if (p.open.load()) did = slice(p);
                    p.inside.fetch_sub(1);
                }
                none = did ? 0 : none + 1;
            }
        }
    }

    const CopyFn fn_;
    Place places_[kPlaces];
    std::atomic<int> sleeping_{0};
    std::atomic<unsigned> copies_{0};
    std::atomic<bool> stop_{false};
    std::mutex mu_;
    std::condition_variable cv_;
    std::vector<std::thread> workers_;  // last: they use what is above
};

}  // namespace iclb
