// The idle-buffer cache of a context (nova_bufcache.h) against a counted stand-in
// for cudaFree: argv[1] names the scenario, the exit status says whether it held.
#include "nova_bufcache.h"

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <thread>

static std::atomic<long> freed{0};

extern "C" cudaError_t cudaFree(void *)
{
    freed++;
    return cudaSuccess;
}

using nova::BufCache;

// host allocation failures on demand
static bool no_memory = false;

__attribute__((noinline)) void *operator new(size_t n)
{
    void *p = no_memory ? nullptr : std::malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
__attribute__((noinline)) void operator delete(void *p) noexcept { std::free(p); }
__attribute__((noinline)) void operator delete(void *p, size_t) noexcept { std::free(p); }

static void *buf(long n) { return reinterpret_cast<void *>(n + 1); }

// buffers put from other threads while the context closes: all are freed
static bool close_race()
{
    for (int round = 0; round < 3000; round++) {
        freed = 0;
        auto cache = std::make_shared<BufCache>();
        long puts = 0;
        for (; puts < 4; puts++) cache->put(buf(puts), 64);
        std::atomic<long> late{0};
        std::atomic<bool> go{false};
        std::thread t[4];
        for (auto &w : t)
            w = std::thread([&] {
                while (!go) {}
                for (int n = 0; n < 200; n++) {
                    cache->put(buf(100), 64);
                    late++;
                }
            });
        go = true;
        while (late < 100) {}
        cache->close();
        for (auto &w : t) w.join();
        cache.reset();
        if (freed != puts + late) {
            std::printf("round %d: %ld buffers, %ld freed\n", round, puts + (long)late, (long)freed);
            return false;
        }
    }
    return true;
}

// the size bound, the reuse by size and the buffers that come back after the close
static bool bound_and_reuse()
{
    freed = 0;
    auto cache = std::make_shared<BufCache>();
    const size_t half = BufCache::kKeep / 2;
    cache->put(buf(0), half);
    cache->put(buf(1), half);
    cache->put(buf(2), half);  // the oldest goes
    bool ok = freed == 1 && cache->take(half) == buf(2) && cache->take(64) == nullptr;
    cache->put(buf(3), BufCache::kKeep + 1);  // too large to keep
    ok = ok && freed == 2;
    cache->put(nullptr, 64);
    cache->close();
    ok = ok && freed == 3;
    cache->put(buf(4), 64);
    return ok && freed == 4 && cache->take(64) == nullptr;
}

// a buffer that the list cannot take for want of host memory is freed, and nothing is thrown
static bool host_memory()
{
    freed = 0;
    auto cache = std::make_shared<BufCache>();
    no_memory = true;
    bool thrown = false;
    try {
        cache->put(buf(0), 64);
    } catch (...) {
        thrown = true;
    }
    no_memory = false;
    return !thrown && freed == 1 && cache->take(64) == nullptr;
}

// a failed allocation gives back the idle buffers of every context and is tried once more
static bool out_of_memory()
{
    freed = 0;
    auto a = std::make_shared<BufCache>(), b = std::make_shared<BufCache>(), gone = std::make_shared<BufCache>();
    int calls = 0;
    auto fails = [&] { return ++calls, 7; };
    bool ok = BufCache::retry(fails) == 7 && calls == 1;  // nothing to give back: no second try
    a->put(buf(0), 64);
    b->put(buf(1), 64);
    gone->put(buf(2), 64);
    gone.reset();
    calls = 0;
    ok = ok && freed == 1 && BufCache::retry([&] { return ++calls, freed == 3 ? 0 : 2; }) == 0 && calls == 2;
    a->put(buf(3), 64);
    calls = 0;
    ok = ok && BufCache::retry([&] { return ++calls, 0; }) == 0 && calls == 1 && freed == 3;
    ok = ok && BufCache::retry(fails) == 7 && calls == 3 && freed == 4;
    return ok && a->take(64) == nullptr && b->take(64) == nullptr;
}

int main(int, char **argv)
{
    if (!std::strcmp(argv[1], "out_of_memory")) return out_of_memory() ? 0 : 1;
    if (!std::strcmp(argv[1], "host_memory")) return host_memory() ? 0 : 1;
    if (!std::strcmp(argv[1], "close_race")) return close_race() ? 0 : 1;
    if (!std::strcmp(argv[1], "bound_and_reuse")) return bound_and_reuse() ? 0 : 1;
    return 2;
}
