// Memory of an engine: a device arena, and page-locked scratch for scalar read-backs.
#pragma once
#include <algorithm>
#include <iterator>
#include <map>
#include <mutex>
#include <vector>

#include "common.cuh"

namespace dnpeff {

// Slabs that engines left when they were destroyed (those that were asked to, option keep_memory), for
// the next engine on the same device: whole jobs from host memory, 300 x 9000 at rank 128 and 8192 x 1048576
// at rank 64 (4 GB of slabs each), take 5.1 and 77 ms without and 4.2 and 62 with it, the
// rest being cudaMalloc and cudaFree.  At most kMost bytes a device, a twentieth of its memory; they go back to the
// device when an allocation here fails, when an engine ends that never needed them, and with dnpeff_release_memory.
class SlabCache {
public:
    static constexpr size_t kMost = (size_t)8 << 30;
    static SlabCache& get() {
        static SlabCache* c = new SlabCache;  // never destroyed: the driver may be gone by then
        return *c;
    }
    // A slab of at least `bytes` and at most a quarter more, or null.
    char* take(int device, size_t bytes, size_t* got) {
        std::lock_guard<std::mutex> lk(mu_);
        auto best = slabs_.end();
        for (auto it = slabs_.begin(); it != slabs_.end(); ++it)
            if (it->device == device && it->bytes >= bytes && it->bytes - it->bytes / 5 <= bytes &&
                (best == slabs_.end() || it->bytes < best->bytes))
                best = it;
        if (best == slabs_.end()) return nullptr;
        char* p = best->p;
        *got = best->bytes;
        slabs_.erase(best);
        return p;
    }
    // Takes an engine's slabs (its stream is idle), small ones first; what does not fit and what
    // lay here all through the engine's life is freed.
    void give(int device, std::vector<std::pair<char*, size_t>> slabs, int64_t born) {
        std::sort(slabs.begin(), slabs.end(), [](auto& a, auto& b) { return a.second < b.second; });
        std::lock_guard<std::mutex> lk(mu_);
        size_t held = 0;
        for (auto it = slabs_.begin(); it != slabs_.end();) {
            if (it->device == device && it->since < born) {
                cudaFree(it->p);
                it = slabs_.erase(it);
            } else {
                if (it->device == device) held += it->bytes;
                ++it;
            }
        }
        for (auto& s : slabs) {
            if (held + s.second <= kMost) {
                slabs_.push_back({device, s.first, s.second, ++clock_});
                held += s.second;
            } else {
                cudaFree(s.first);
            }
        }
    }
    void flush(int device) {  // (-1: of every device)
        std::lock_guard<std::mutex> lk(mu_);
        for (auto it = slabs_.begin(); it != slabs_.end();) {
            if (device < 0 || it->device == device) {
                cudaFree(it->p);
                it = slabs_.erase(it);
            } else {
                ++it;
            }
        }
    }
    size_t held(int device) {
        std::lock_guard<std::mutex> lk(mu_);
        size_t n = 0;
        for (auto& s : slabs_)
            if (s.device == device) n += s.bytes;
        return n;
    }
    int64_t now() {
        std::lock_guard<std::mutex> lk(mu_);
        return ++clock_;
    }

private:
    struct Slab {
        int device;
        char* p;
        size_t bytes;
        int64_t since;
    };
    std::mutex mu_;
    std::vector<Slab> slabs_;
    int64_t clock_ = 0;
};

// Idle streams of engines that were destroyed, for the next ones (making and destroying one takes 0.3 ms).
class StreamCache {
public:
    static constexpr size_t kMost = 8;
    static StreamCache& get() {
        static StreamCache* c = new StreamCache;  // never destroyed: the driver may be gone by then
        return *c;
    }
    cudaError_t take(int device, cudaStream_t* out) {  // with the device current
        {
            std::lock_guard<std::mutex> lk(mu_);
            for (auto it = idle_.begin(); it != idle_.end(); ++it)
                if (it->first == device) {
                    *out = it->second;
                    idle_.erase(it);
                    return cudaSuccess;
                }
        }
        return cudaStreamCreateWithFlags(out, cudaStreamNonBlocking);
    }
    void flush(int device) {  // (-1: of every device)
        std::lock_guard<std::mutex> lk(mu_);
        for (auto it = idle_.begin(); it != idle_.end();) {
            if (device < 0 || it->first == device) {
                cudaStreamDestroy(it->second);
                it = idle_.erase(it);
            } else {
                ++it;
            }
        }
    }
    void give(int device, cudaStream_t st) {
        if (cudaStreamSynchronize(st) == cudaSuccess) {
            std::lock_guard<std::mutex> lk(mu_);
            if (idle_.size() < kMost) {
                idle_.push_back({device, st});
                return;
            }
        }
        cudaStreamDestroy(st);
    }

private:
    std::mutex mu_;
    std::vector<std::pair<int, cudaStream_t>> idle_;
};

// Device memory of one engine.  A cudaMalloc or cudaFree that reaches the driver's memory manager
// takes 0.35 ms on a quiet host and 2.2 ms on a busy one, whatever its size up to 256 MB (only
// requests up to 1 MB share a chunk and mostly take 3 microseconds); the loader makes some fifty
// allocations and a small matrix is loaded in well under a millisecond of kernels.  Here they
// come from slabs that stay with the engine, so that a load makes one or a few such calls, and
// none when the engine is loaded again (row chunks of a coefficient fit).  Two classes: blocks
// below kSlab are cut from shared slabs of that size, best fit, coalesced when freed; larger ones
// are slabs of their own, reused whole by a request of at least four fifths of their size.  Reuse
// is ordered by the engine's stream: everything that touches a block runs on it, or on a stream
// that waits for it first.
class DeviceArena {
public:
    static constexpr size_t kSlab = (size_t)64 << 20;
    static constexpr size_t kKeep = (size_t)2 << 30;  // unused bytes that stay after a load

    DeviceArena() {}
    DeviceArena(const DeviceArena&) = delete;
    DeviceArena& operator=(const DeviceArena&) = delete;

    // `st`: the engine's stream, waited for before memory goes back to the device.
    void open(int device, cudaStream_t st) {
        device_ = device;
        st_ = st;
        born_ = SlabCache::get().now();
    }

    int alloc(size_t bytes, void** out) {
        bytes = (std::max<size_t>(bytes, 1) + 511) / 512 * 512;
        const bool own = bytes >= kSlab;
        auto best = slabs_.end();
        size_t best_off = 0, best_len = SIZE_MAX;
        for (auto it = slabs_.begin(); it != slabs_.end(); ++it) {
            Slab& s = it->second;
            if (s.own != own) continue;
            if (own) {
                if (s.used == 0 && s.bytes >= bytes && s.bytes - s.bytes / 5 <= bytes && s.bytes < best_len) {
                    best = it;
                    best_len = s.bytes;
                }
                continue;
            }
            for (auto& f : s.free)
                if (f.second >= bytes && f.second < best_len) {
                    best = it;
                    best_off = f.first;
                    best_len = f.second;
                }
        }
        if (best == slabs_.end()) {
            size_t want = own ? (bytes + ((size_t)2 << 20) - 1) >> 21 << 21 : kSlab;
            void* p = SlabCache::get().take(device_, want, &want);
            cudaError_t e = p ? cudaSuccess : cudaMalloc(&p, want);
            if (e == cudaErrorMemoryAllocation) {  // give back what lies unused and try once more
                cudaGetLastError();
                trim(0);
                SlabCache::get().flush(device_);
                e = cudaMalloc(&p, want);
            }
            if (e != cudaSuccess) {
                cudaGetLastError();
                return fail(DNPEFF_ERR_CUDA, "cudaMalloc of %zu bytes: %s", want, cudaGetErrorString(e));
            }
            best = slabs_.emplace((char*)p, Slab()).first;
            best->second.bytes = want;
            best->second.own = own;
            best->second.free[0] = want;
            best_len = want;
        }
        Slab& s = best->second;
        s.free.erase(best_off);
        const size_t take = own ? best_len : bytes;
        if (best_len > take) s.free[best_off + take] = best_len - take;
        s.used += take;
        live_[best->first + best_off] = {take, bytes};
        asked_ += bytes;
        *out = best->first + best_off;
        return DNPEFF_OK;
    }

    void release(void* p) {
        auto it = live_.find((char*)p);
        if (it == live_.end()) return;
        size_t len = it->second.first;
        asked_ -= it->second.second;
        live_.erase(it);
        auto sl = std::prev(slabs_.upper_bound((char*)p));
        Slab& s = sl->second;
        const size_t off = (size_t)((char*)p - sl->first);
        s.used -= len;
        auto next = s.free.lower_bound(off);
        if (next != s.free.end() && off + len == next->first) {
            len += next->second;
            next = s.free.erase(next);
        }
        if (next != s.free.begin()) {
            auto prev = std::prev(next);
            if (prev->first + prev->second == off) {
                prev->second += len;
                return;
            }
        }
        s.free[off] = len;
    }

    // Bytes of slabs without a live block.
    size_t unused() const {
        size_t n = 0;
        for (auto& kv : slabs_)
            if (kv.second.used == 0) n += kv.second.bytes;
        return n;
    }

    // Memory that the engine may plan with: what the device has free, and what lies in the engine's slabs and in
    // those that other engines left beyond what live blocks asked for.  The same for the same load whatever
    // slabs there are from earlier ones, so that sizes derived from it (and with them the order of sums) do not
    // depend on a process's history.  What others hold counts; to five leading bits, so
    // that a module loaded meanwhile hardly ever does.
    int at_hand(size_t* out) const {
        size_t free_b = 0, total_b = 0;
        DN_CUDA(cudaMemGetInfo(&free_b, &total_b));
        for (auto& kv : slabs_) free_b += kv.second.bytes;
        free_b += SlabCache::get().held(device_);
        free_b -= std::min(free_b, asked_);
        size_t unit = 1;
        while (free_b / unit >= 32) unit *= 2;
        *out = free_b / unit * unit;
        return DNPEFF_OK;
    }

    // Slabs without a live block go back to the device until at most `keep` unused bytes are left.
    void trim(size_t keep) {
        size_t left = unused();
        bool waited = false;
        while (left > keep) {
            auto big = slabs_.end();
            for (auto it = slabs_.begin(); it != slabs_.end(); ++it)
                if (it->second.used == 0 && (big == slabs_.end() || it->second.bytes > big->second.bytes)) big = it;
            if (big == slabs_.end()) break;
            if (!waited && st_) cudaStreamSynchronize(st_);
            waited = true;
            cudaFree(big->first);
            left -= big->second.bytes;
            slabs_.erase(big);
        }
    }

    // Everything goes, live or not (the engine is being destroyed, its streams are idle): to the next engine
    // (keep) or to the device.
    void close(bool keep) {
        std::vector<std::pair<char*, size_t>> all;
        for (auto& kv : slabs_) {
            if (keep) all.push_back({kv.first, kv.second.bytes});
            else cudaFree(kv.first);
        }
        if (keep) SlabCache::get().give(device_, std::move(all), born_);
        slabs_.clear();
        live_.clear();
        asked_ = 0;
    }

private:
    struct Slab {
        size_t bytes = 0, used = 0;
        bool own = false;
        std::map<size_t, size_t> free;  // offset -> length
    };
    std::map<char*, Slab> slabs_;
    std::map<char*, std::pair<size_t, size_t>> live_;  // length, and what was asked for
    size_t asked_ = 0;
    cudaStream_t st_ = nullptr;
    int device_ = 0;
    int64_t born_ = 0;
};

// The arena that DevBuf uses on this thread (that of the engine whose call is being made).
inline DeviceArena*& current_arena() {
    static thread_local DeviceArena* a = nullptr;
    return a;
}
struct ArenaScope {
    DeviceArena* saved;
    explicit ArenaScope(DeviceArena* a) : saved(current_arena()) { current_arena() = a; }
    ~ArenaScope() { current_arena() = saved; }
};

// Device memory for the length of a scope: from the engine's arena, or from cudaMalloc in calls
// that have no engine.
template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t count = 0;
    DeviceArena* arena = nullptr;
    DevBuf() {}
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    int alloc(size_t n) {
        release();
        count = n;
        arena = current_arena();
        if (arena) return arena->alloc(sizeof(T) * n, (void**)&p);
        DN_CUDA(cudaMalloc((void**)&p, sizeof(T) * (n ? n : 1)));
        return DNPEFF_OK;
    }
    int alloc_zero(size_t n, cudaStream_t st) {
        DN_TRY(alloc(n));
        DN_CUDA(cudaMemsetAsync(p, 0, sizeof(T) * (n ? n : 1), st));
        return DNPEFF_OK;
    }
    void release() {
        if (p) {
            if (arena) arena->release(p);
            else cudaFree(p);
        }
        p = nullptr;
        count = 0;
    }
};

// Page-locked scratch of one engine (kPinnedBytes): slots of one page-locked block that the
// process keeps (256 KB), since making such a block takes longer than loading a small matrix.
// Engines beyond the number of slots make their own.
constexpr size_t kPinnedBytes = 8192;
class PinnedSlots {
public:
    static PinnedSlots& get() {
        static PinnedSlots* s = new PinnedSlots;  // never destroyed: the driver may be gone by then
        return *s;
    }
    void* take() {
        std::lock_guard<std::mutex> lk(mu_);
        if (!block_ && !tried_) {
            tried_ = true;
            if (cudaHostAlloc((void**)&block_, kPinnedBytes * kSlots, cudaHostAllocPortable) != cudaSuccess) {
                cudaGetLastError();
                block_ = nullptr;
            }
        }
        for (int i = 0; block_ && i < kSlots; i++)
            if (!used_[i]) {
                used_[i] = true;
                return block_ + (size_t)i * kPinnedBytes;
            }
        void* p = nullptr;
        if (cudaHostAlloc(&p, kPinnedBytes, cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        return p;
    }
    void give(void* p) {
        if (!p) return;
        std::lock_guard<std::mutex> lk(mu_);
        if (block_ && (char*)p >= block_ && (char*)p < block_ + kPinnedBytes * kSlots)
            used_[(size_t)((char*)p - block_) / kPinnedBytes] = false;
        else
            cudaFreeHost(p);
    }

private:
    static constexpr int kSlots = 32;
    std::mutex mu_;
    char* block_ = nullptr;
    bool tried_ = false;
    bool used_[kSlots] = {false};
};

}  // namespace dnpeff
