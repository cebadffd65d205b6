// Device-to-host copies of large results into pageable memory.
//
// A plain cudaMemcpyAsync to pageable memory is one thread's work in the driver:
// it stages, copies and, in memory that the caller has just allocated, takes a
// page fault every 4 KiB (99 MB of arrivals: 22-27 ms, 4 GB/s). Here the copy
// engine fills a ring of pinned chunks and a few threads empty it, so faults and
// copies run in parallel beside the transfer: 8-10 ms. The ring (4 MB) belongs to
// one context and is given back with it. Making it takes 4-5 ms, once, so results
// below 32 MB, for which the first copy would lose by it, go the plain way.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>
#include <vector>

namespace bhcb {

class HostCopy {
public:
    HostCopy() = default;
    HostCopy(const HostCopy &) = delete;
    HostCopy &operator=(const HostCopy &) = delete;
    ~HostCopy() { release(); }

    // Copies after the work queued on st. The plain copy for small results and for
    // memory that CUDA knows; the caller synchronises st as after any asynchronous
    // copy.
    cudaError_t copy(void *dst, const void *src, size_t bytes, cudaStream_t st)
    {
        if(bytes < MIN_BYTES || !pageable(dst) || !prepare())
            return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
        int device = 0;
        cudaError_t err = cudaGetDevice(&device);
        if(err != cudaSuccess) return err;
        const long long n = (long long)((bytes + CHUNK - 1) / CHUNK);
        std::atomic<long long> issued{0}, taken{0};
        std::atomic<bool> failed{false};
        for(auto &d : done_) d.store(-1, std::memory_order_relaxed);
        auto work = [&]() {
            cudaSetDevice(device);
            for(;;) {
                const long long i = taken.fetch_add(1);
                if(i >= n) return;
                while(issued.load(std::memory_order_acquire) <= i) {
                    if(failed.load()) return;
                    std::this_thread::yield();
                }
                const int s = (int)(i % SLOTS);
                if(cudaEventSynchronize(ev_[s]) != cudaSuccess) {
                    failed.store(true);
                    return;
                }
                const size_t off = (size_t)i * CHUNK;
                std::memcpy((char *)dst + off, ring_ + (size_t)s * CHUNK, std::min<size_t>(CHUNK, bytes - off));
                done_[s].store(i, std::memory_order_release);
            }
        };
        const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
        const int nt = (int)std::min<unsigned>(MAX_THREADS, cores);
        std::vector<std::thread> threads;
        try {
            for(int t = 0; t < nt; ++t) threads.emplace_back(work);
        } catch(...) {   // no more threads: those there are do it
        }
        if(threads.empty()) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
        for(long long i = 0; i < n && !failed.load(); ++i) {
            const int s = (int)(i % SLOTS);
            while(i >= SLOTS && done_[s].load(std::memory_order_acquire) != i - SLOTS && !failed.load())
                std::this_thread::yield();
            const size_t off = (size_t)i * CHUNK;
            err = cudaMemcpyAsync(ring_ + (size_t)s * CHUNK, (const char *)src + off, std::min<size_t>(CHUNK, bytes - off),
                                  cudaMemcpyDeviceToHost, st);
            if(err == cudaSuccess) err = cudaEventRecord(ev_[s], st);
            if(err != cudaSuccess) {
                failed.store(true);
                break;
            }
            issued.store(i + 1, std::memory_order_release);
        }
        for(auto &t : threads) t.join();
        if(err == cudaSuccess && failed.load()) {
            err = cudaStreamSynchronize(st);
            if(err == cudaSuccess) err = cudaErrorUnknown;
        }
        return err;
    }

    void release()
    {
        for(auto &e : ev_)
            if(e) cudaEventDestroy(e);
        for(auto &e : ev_) e = nullptr;
        if(ring_) cudaFreeHost(ring_);
        ring_ = nullptr;
    }

private:
    static constexpr size_t CHUNK = 512u << 10, MIN_BYTES = 32u << 20;
    static constexpr int SLOTS = 8, MAX_THREADS = 8;
    char *ring_ = nullptr;
    cudaEvent_t ev_[SLOTS] = {};
    std::atomic<long long> done_[SLOTS];   // last chunk copied out of each slot

    // Errors of the two probes below are taken back, so that the caller does not find
    // them; an error from before the copy is left for whoever asks for it.
    static bool pageable(const void *p)
    {
        cudaPointerAttributes at{};
        if(cudaPointerGetAttributes(&at, p) == cudaSuccess) return at.type == cudaMemoryTypeUnregistered;
        cudaGetLastError();
        return false;
    }
    bool prepare()
    {
        if(ring_) return true;
        void *p = nullptr;
        bool ok = cudaHostAlloc(&p, CHUNK * SLOTS, cudaHostAllocDefault) == cudaSuccess;
        ring_ = ok ? (char *)p : nullptr;
        for(auto &e : ev_) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
        if(!ok) {
            cudaGetLastError();
            release();
        }
        return ok;
    }
};

} // namespace bhcb
