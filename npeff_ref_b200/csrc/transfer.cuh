// Copies between the caller's host arrays and the device.
//
// The driver moves pageable memory through one staging buffer filled by one thread: about
// 10 GB/s up and 5 GB/s down (where the pages of a fresh result array are also faulted in by that
// thread), against 55 GB/s for page-locked memory.  Large pageable arrays therefore go through a
// ring of page-locked chunks filled, or emptied, by several host threads; page-locked and small
// arrays are handed to cudaMemcpyAsync as they are.
#pragma once
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include "common.cuh"

namespace dnpeff {

inline bool host_pageable(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// The process's page-locked chunks: kThreads threads, two chunks each (32 MB, made on first use
// and kept until dnpeff_release_memory: page-locking them takes as long as moving several hundred MB).  One transfer at a
// time holds them; whoever finds them taken copies the plain way.
struct StagingRing {
    static constexpr int kThreads = 8;
    static constexpr size_t kChunk = (size_t)2 << 20;
    std::mutex mu;
    char* base = nullptr;

    static StagingRing& get() {
        static StagingRing* r = new StagingRing;  // never destroyed: the driver may be gone by then
        return *r;
    }
    bool ready() {  // with mu held
        if (!base && cudaHostAlloc((void**)&base, 2 * kThreads * kChunk, cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            base = nullptr;
        }
        return base != nullptr;
    }
    void release() {  // unless a transfer holds them
        std::unique_lock<std::mutex> lk(mu, std::try_to_lock);
        if (!lk.owns_lock() || !base) return;
        cudaFreeHost(base);
        base = nullptr;
    }
    // Threads worth starting for that many bytes (starting one costs about what it takes to copy
    // a quarter of a megabyte), and the bytes that one handles at a time.
    static int threads_for(size_t bytes, int most = kThreads) {
        const size_t cores = std::max(1u, std::thread::hardware_concurrency());
        return (int)std::min<size_t>(bytes >> 20, std::min<size_t>((size_t)most, cores));
    }
    static size_t chunk_for(size_t bytes, int threads) {
        const size_t even = (bytes / (4 * (size_t)threads) + 65535) >> 16 << 16;
        return std::min(kChunk, std::max<size_t>(even, (size_t)256 << 10));
    }
};

// An upload of several parts, in order, on one stream.  Part p has been handed to the stream once
// wait(p) returns, which also makes another stream wait for its arrival.  The destructor joins
// the threads and waits for the copies.
class Upload {
public:
    struct Part {
        void* dst;
        const void* src;
        size_t bytes;
    };

    ~Upload() {
        for (auto& t : threads_) t.join();
        if (st_) cudaStreamSynchronize(st_);
        for (cudaEvent_t e : ready_)
            if (e) cudaEventDestroy(e);
        if (held_) StagingRing::get().mu.unlock();
    }

    int start(std::vector<Part> parts, int device, cudaStream_t st) {
        parts_ = std::move(parts);
        st_ = st;
        size_t total = 0;
        bool pageable = false;
        for (const Part& p : parts_) total += p.bytes;
        ready_.assign(parts_.size(), nullptr);
        left_.reset(new std::atomic<int64_t>[std::max<size_t>(parts_.size(), 1)]);
        issued_.assign(parts_.size(), 0);
        for (cudaEvent_t& e : ready_) DN_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        const int n_threads = StagingRing::threads_for(total);
        if (n_threads >= 2)
            for (const Part& p : parts_) pageable = pageable || (p.bytes > 0 && host_pageable(p.src));
        if (pageable) held_ = StagingRing::get().mu.try_lock();
        if (!held_ || !StagingRing::get().ready()) {
            for (size_t p = 0; p < parts_.size(); p++) {
                if (parts_[p].bytes)
                    DN_CUDA(cudaMemcpyAsync(parts_[p].dst, parts_[p].src, parts_[p].bytes, cudaMemcpyHostToDevice, st));
                DN_CUDA(cudaEventRecord(ready_[p], st));
                issued_[p] = 1;
            }
            return DNPEFF_OK;
        }
        chunk_ = StagingRing::chunk_for(total, n_threads);
        for (size_t p = 0; p < parts_.size(); p++) {
            const int64_t chunks = (int64_t)((parts_[p].bytes + chunk_ - 1) / chunk_);
            left_[p] = chunks;
            first_.push_back(n_chunks_);
            n_chunks_ += chunks;
            if (chunks == 0) {
                DN_CUDA(cudaEventRecord(ready_[p], st));
                issued_[p] = 1;
            }
        }
        try {
            for (int t = 0; t < n_threads; t++) threads_.emplace_back([this, t, device] { work(t, device); });
        } catch (const std::system_error&) {  // no more threads to be had: those that started do it all
            if (threads_.empty()) work(0, device);
        }
        return DNPEFF_OK;
    }

    int wait(size_t p, cudaStream_t st) {
        {
            std::unique_lock<std::mutex> lk(mu_);
            cv_.wait(lk, [&] { return issued_[p] != 0; });
        }
        if (error_.load() != (int)cudaSuccess)
            return fail(DNPEFF_ERR_CUDA, "upload: %s", cudaGetErrorString((cudaError_t)error_.load()));
        DN_CUDA(cudaStreamWaitEvent(st, ready_[p], 0));
        return DNPEFF_OK;
    }

private:
    void work(int t, int device) {
        cudaError_t e = cudaSetDevice(device);
        char* const slots = StagingRing::get().base + (size_t)t * 2 * StagingRing::kChunk;
        cudaEvent_t done[2] = {nullptr, nullptr};
        for (cudaEvent_t& d : done)
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&d, cudaEventDisableTiming);
        for (int k = 0;; k++) {
            const int64_t c = next_.fetch_add(1);
            if (c >= n_chunks_) break;
            const size_t p = (size_t)(std::upper_bound(first_.begin(), first_.end(), c) - first_.begin()) - 1;
            const size_t off = (size_t)(c - first_[p]) * chunk_;
            const size_t n = std::min(chunk_, parts_[p].bytes - off);
            char* slot = slots + (size_t)(k & 1) * StagingRing::kChunk;
            if (e == cudaSuccess && k >= 2) e = cudaEventSynchronize(done[k & 1]);
            if (e == cudaSuccess) {
                memcpy(slot, (const char*)parts_[p].src + off, n);
                e = cudaMemcpyAsync((char*)parts_[p].dst + off, slot, n, cudaMemcpyHostToDevice, st_);
            }
            if (e == cudaSuccess) e = cudaEventRecord(done[k & 1], st_);
            if (e != cudaSuccess) error_ = (int)e;
            if (left_[p].fetch_sub(1) == 1) {  // the part's last chunk is in the stream
                cudaEventRecord(ready_[p], st_);
                std::lock_guard<std::mutex> lk(mu_);
                issued_[p] = 1;
                cv_.notify_all();
            }
        }
        for (cudaEvent_t d : done)
            if (d) {
                cudaEventSynchronize(d);  // the chunk may be another transfer's afterwards
                cudaEventDestroy(d);
            }
    }

    std::vector<Part> parts_;
    std::vector<cudaEvent_t> ready_;
    std::unique_ptr<std::atomic<int64_t>[]> left_;
    std::vector<char> issued_;
    std::vector<int64_t> first_;
    size_t chunk_ = StagingRing::kChunk;
    int64_t n_chunks_ = 0;
    std::atomic<int64_t> next_{0};
    std::atomic<int> error_{(int)cudaSuccess};
    std::mutex mu_;
    std::condition_variable cv_;
    std::vector<std::thread> threads_;
    cudaStream_t st_ = nullptr;
    bool held_ = false;
};

// Device -> host behind the work queued on `st`; returns when the bytes are there.
// Twice as many threads on chunks of half the size: they also fault in the pages of a fresh result
// array (268 MB: 11.3 -> 9.8 ms; an upload has its limit in eight, 12.7 -> 14.2 ms for 537 MB with sixteen).
inline int download(void* dst, const void* src, size_t bytes, int device, cudaStream_t st) {
    constexpr size_t kSlot = StagingRing::kChunk / 2;
    const int n_threads = StagingRing::threads_for(bytes, 2 * StagingRing::kThreads);
    StagingRing& ring = StagingRing::get();
    std::unique_lock<std::mutex> lk(ring.mu, std::defer_lock);
    if (n_threads < 2 || !host_pageable(dst) || !lk.try_lock() || !ring.ready()) {
        if (bytes) DN_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
        DN_CUDA(cudaStreamSynchronize(st));
        return DNPEFF_OK;
    }
    const size_t chunk = std::min(kSlot, StagingRing::chunk_for(bytes, n_threads));
    const int64_t n_chunks = (int64_t)((bytes + chunk - 1) / chunk);
    std::atomic<int64_t> next{0};
    std::atomic<int> error{(int)cudaSuccess};
    auto work = [&](int t) {
        cudaError_t e = cudaSetDevice(device);
        char* const slots = ring.base + (size_t)t * 2 * kSlot;
        cudaEvent_t done[2] = {nullptr, nullptr};
        for (cudaEvent_t& d : done)
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&d, cudaEventDisableTiming);
        int64_t held[2] = {-1, -1};
        auto ask = [&](int s) {
            held[s] = -1;
            const int64_t c = next.fetch_add(1);
            if (c >= n_chunks || e != cudaSuccess) return;
            const size_t off = (size_t)c * chunk, n = std::min(chunk, bytes - off);
            e = cudaMemcpyAsync(slots + (size_t)s * kSlot, (const char*)src + off, n, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaEventRecord(done[s], st);
            held[s] = c;
        };
        ask(0);
        ask(1);
        for (int s = 0; held[s] >= 0; s ^= 1) {
            if (e == cudaSuccess) e = cudaEventSynchronize(done[s]);
            if (e != cudaSuccess) break;
            const size_t off = (size_t)held[s] * chunk;
            memcpy((char*)dst + off, slots + (size_t)s * kSlot, std::min(chunk, bytes - off));
            ask(s);
        }
        if (e != cudaSuccess) error = (int)e;
        for (cudaEvent_t d : done)
            if (d) cudaEventDestroy(d);
    };
    std::vector<std::thread> threads;
    try {
        for (int t = 1; t < n_threads; t++) threads.emplace_back(work, t);
    } catch (const std::system_error&) {  // fewer threads share the chunks
    }
    work(0);
    for (auto& t : threads) t.join();
    DN_CUDA(cudaStreamSynchronize(st));
    if (error.load() != (int)cudaSuccess)
        return fail(DNPEFF_ERR_CUDA, "read-back: %s", cudaGetErrorString((cudaError_t)error.load()));
    return DNPEFF_OK;
}

}  // namespace dnpeff
