// Device buffers of dropped fields and matrices that a context keeps for its
// next ones, by size.  Host code only (tests/cpp/bufcache_driver.cpp runs it
// against a stand-in for cudaFree).
#pragma once

#include <cuda_runtime_api.h>

#include <algorithm>
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
// At most kKeep bytes stay (the oldest go first).  All go when the context is
// destroyed, after which buffers still held by fields or matrices are freed
// directly, and when an allocation or an FFT plan of any context in the process
// fails, which is then tried again (retry).
class BufCache {
public:
    static constexpr size_t kKeep = size_t(1) << 30;
    BufCache()
    {
        Live &r = live();
        std::lock_guard<std::mutex> l(r.mu);
        r.all.push_back(this);
    }
    BufCache(const BufCache &) = delete;
    ~BufCache()
    {
        {
            Live &r = live();
            std::lock_guard<std::mutex> l(r.mu);
            r.all.erase(std::find(r.all.begin(), r.all.end(), this));
        }
        trim();
    }
    // make() -> 0 or an error code; after an error the idle buffers of every
    // context go back to the device, and if there were any it is called once more
    template <class Make> static auto retry(Make &&make) -> decltype(make())
    {
        auto e = make();
        return static_cast<int>(e) != 0 && trim_all() ? make() : e;
    }
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
    bool trim()  // whether there was anything to free
    {
        std::lock_guard<std::mutex> l(mu_);
        const bool any = !idle_.empty();
        while (!idle_.empty()) drop();
        return any;
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
    struct Live {  // the caches of the process; never destroyed: contexts may outlive static objects
        std::mutex mu;
        std::vector<BufCache *> all;
    };
    static Live &live()
    {
        static Live *r = new Live;
        return *r;
    }
    static bool trim_all()
    {
        Live &r = live();
        std::lock_guard<std::mutex> l(r.mu);
        bool any = false;
        for (BufCache *c : r.all) any = c->trim() || any;
        return any;
    }
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
