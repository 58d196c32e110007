// Device allocation, and the device buffers that calls keep for one another.
#pragma once

#include <cuda_runtime.h>
#include <atomic>
#include <mutex>
#include <utility>
#include <vector>

namespace vgh {

// Device allocations and frees made by this library since it was loaded (all of them go through device_alloc(),
// DevBuf and TempPool), readable through vg_debug_allocations.
inline std::atomic<uint64_t> g_mallocs{0}, g_frees{0};

// Device buffers that entry points use for the length of a call (rays and hits, records, AOV planes), kept
// for the next call: a cudaMalloc and cudaFree of some tens of MB cost more than most of those calls'
// kernels. A buffer has one owner at a time (TempBuf), whichever thread that is on. All of its uses are in the
// order of the context's stream, so that the next owner's work comes after the last one's. At most KEEP bytes
// wait here (twice that while the stream is busy: freeing waits for the GPU); they go with the context, or when
// an allocation on the device finds no room (device_alloc).
struct TempPool {
    static constexpr size_t KEEP = 256u << 20;
    const int device;
    std::mutex mu;
    std::vector<std::pair<void*, size_t>> idle;
    size_t idle_bytes = 0;

    explicit TempPool(int dev) : device(dev)
    {
        std::lock_guard<std::mutex> lock(all_mu());
        all().push_back(this);
    }
    TempPool(const TempPool&) = delete;
    TempPool& operator=(const TempPool&) = delete;
    ~TempPool()
    {
        {
            std::lock_guard<std::mutex> lock(all_mu());
            for (size_t i = 0; i < all().size(); i++)
                if (all()[i] == this) {
                    all().erase(all().begin() + (long)i);
                    break;
                }
        }
        free_idle();
    }
    // The smallest idle buffer of at least n bytes and at most four times that.
    void* take(size_t n, size_t* bytes)
    {
        std::lock_guard<std::mutex> lock(mu);
        size_t best = idle.size();
        for (size_t i = 0; i < idle.size(); i++)
            if (idle[i].second >= n && idle[i].second / 4 <= n && (best == idle.size() || idle[i].second < idle[best].second))
                best = i;
        if (best == idle.size())
            return nullptr;
        void* p = idle[best].first;
        *bytes = idle[best].second;
        idle_bytes -= idle[best].second;
        idle.erase(idle.begin() + (long)best);
        return p;
    }
    void give(void* p, size_t bytes, cudaStream_t s)
    {
        std::vector<void*> drop;
        {
            std::lock_guard<std::mutex> lock(mu);
            size_t keep = KEEP;
            if (idle_bytes + bytes > KEEP && cudaStreamQuery(s) == cudaErrorNotReady)
                keep = 2 * KEEP;
            if (bytes <= keep) {
                while (idle_bytes + bytes > keep) { // the oldest first
                    drop.push_back(idle.front().first);
                    idle_bytes -= idle.front().second;
                    idle.erase(idle.begin());
                }
                idle.emplace_back(p, bytes);
                idle_bytes += bytes;
            } else {
                drop.push_back(p);
            }
        }
        for (void* q : drop) {
            cudaFree(q);
            g_frees++;
        }
    }
    // Frees what waits here; says how many bytes that was.
    size_t free_idle()
    {
        std::vector<std::pair<void*, size_t>> drop;
        size_t bytes;
        {
            std::lock_guard<std::mutex> lock(mu);
            drop.swap(idle);
            bytes = idle_bytes;
            idle_bytes = 0;
        }
        for (auto& b : drop) {
            cudaFree(b.first);
            g_frees++;
        }
        return bytes;
    }
    // The same for all contexts of a device.
    static size_t free_idle_on(int dev)
    {
        std::lock_guard<std::mutex> lock(all_mu());
        size_t bytes = 0;
        for (TempPool* p : all())
            if (p->device == dev)
                bytes += p->free_idle();
        return bytes;
    }

private:
    static std::mutex& all_mu()
    {
        static std::mutex* m = new std::mutex; // (never destroyed: a context may end after the statics)
        return *m;
    }
    static std::vector<TempPool*>& all()
    {
        static std::vector<TempPool*>* v = new std::vector<TempPool*>;
        return *v;
    }
};

// Device memory of n bytes on the current device. Where it finds no room, the device's idle buffers go and it
// looks once more. *available: the free memory at the last look.
inline cudaError_t device_alloc(void** p, size_t n, size_t* available)
{
    for (bool again = false;; again = true) {
        *p = nullptr;
        size_t total = 0;
        cudaError_t e = cudaMemGetInfo(available, &total);
        if (e != cudaSuccess)
            return e;
        e = n > *available ? cudaErrorMemoryAllocation : cudaMalloc(p, n);
        if (e == cudaSuccess) {
            g_mallocs++;
            return e;
        }
        *p = nullptr;
        int dev = 0;
        if (e != cudaErrorMemoryAllocation || again || cudaGetDevice(&dev) != cudaSuccess || TempPool::free_idle_on(dev) == 0)
            return e;
        cudaGetLastError(); // (the failed attempt's)
    }
}

} // namespace vgh
