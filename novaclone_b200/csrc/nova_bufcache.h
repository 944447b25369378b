// Device buffers of dropped fields and matrices that a context keeps for its
// next ones, by size.  Host code only (tests/cpp/bufcache_driver.cpp runs it
// against a stand-in for cudaFree).
#pragma once

#include <cuda_runtime_api.h>

#include <memory>
#include <mutex>
#include <new>
#include <utility>
#include <vector>

namespace nova {

// The reference's explicit programs make and drop a field
// per operator call (ex::grad, ex::div, ...); with a cudaMalloc and a cudaFree
// each (about 0.35 + 0.3 ms) the operator calls of a 128^3 step took 5.5 ms
// around 1.3 ms of kernels, now 1.4 ms.  A buffer is put here only after the
// work that uses it has been waited for (nova_field_destroy, nova_fdm_destroy).
// At most kKeep bytes stay (the oldest go first); all go when an allocation
// fails or the context is destroyed, after which buffers still held by fields
// or matrices are freed directly.
class BufCache {
public:
    static constexpr size_t kKeep = size_t(1) << 30;
    BufCache() = default;
    BufCache(const BufCache &) = delete;
    ~BufCache() { trim(); }
    void *take(size_t bytes)
    {
        std::lock_guard<std::mutex> l(mu_);
        for (size_t q = idle_.size(); q-- > 0;)
            if (idle_[q].second == bytes) {
                void *p = idle_[q].first;
                held_ -= bytes;
                idle_.erase(idle_.begin() + q);
                return p;
            }
        return nullptr;
    }
    void put(void *p, size_t bytes)
    {
        if (!p) return;
        std::lock_guard<std::mutex> l(mu_);
        if (!open_ || bytes > kKeep) {
            cudaFree(p);
            return;
        }
        while (held_ + bytes > kKeep) drop();
        try {
            idle_.emplace_back(p, bytes);
        } catch (const std::bad_alloc &) {  // the callers are C entry points
            cudaFree(p);
            return;
        }
        held_ += bytes;
    }
    void trim()
    {
        std::lock_guard<std::mutex> l(mu_);
        while (!idle_.empty()) drop();
    }
    // from here on put() frees (set under the lock that empties the list: a
    // buffer put between the two would stay allocated for good)
    void close()
    {
        std::lock_guard<std::mutex> l(mu_);
        open_ = false;
        while (!idle_.empty()) drop();
    }

private:
    void drop()
    {
        cudaFree(idle_.front().first);
        held_ -= idle_.front().second;
        idle_.erase(idle_.begin());
    }
    std::mutex mu_;
    std::vector<std::pair<void *, size_t>> idle_;
    size_t held_ = 0;
    bool open_ = true;
};

}  // namespace nova
