// The plans' device memory (csrc/dcpse_memory.h) over a fake runtime: a block is
// handed out again only after a wait later than its release, the wait is a
// cudaFree (nothing that a capture elsewhere forbids is called), a refused
// allocation gives the free blocks back and leaves no error behind.
#include <cstdio>
#include <cstdint>
#include <map>
#include <random>
#include <set>
#include <thread>

#include "dcpse_memory.h"

#define CHECK(c)                                                    \
    do {                                                            \
        if (!(c)) {                                                 \
            std::printf("%s:%d: %s\n", __FILE__, __LINE__, #c);     \
            return 1;                                               \
        }                                                           \
    } while (0)

struct Fake {
    typedef int Error;
    static constexpr int ok = 0, no_memory = 2;
    static std::mutex m;
    static std::map<void*, size_t> blocks;  // of the driver
    static size_t used, limit;
    static int dev, last_error, frees;
    static bool refuse;                     // as under a global-mode capture
    static bool broken;                     // no allocation at all
    static thread_local bool relaxed;
    struct Relaxed {
        Relaxed() { relaxed = true; }
        ~Relaxed() { relaxed = false; }
    };
    static uintptr_t next;
    static int malloc(void** p, size_t bytes) {
        std::lock_guard<std::mutex> lock(m);
        *p = nullptr;
        if (broken || (refuse && !relaxed)) return last_error = 900;
        if (bytes > limit - used) return last_error = no_memory;
        used += bytes;
        *p = reinterpret_cast<void*>(next);
        next += bytes + 256;
        blocks[*p] = bytes;
        return ok;
    }
    static int free(void* p) {
        std::lock_guard<std::mutex> lock(m);
        if (refuse && !relaxed) return last_error = 900;
        auto it = blocks.find(p);
        if (it == blocks.end()) return last_error = 1;
        used -= it->second;
        blocks.erase(it);
        ++frees;
        return ok;
    }
    static int device(int* d) {
        *d = dev;
        return ok;
    }
    static void clear_error() { last_error = 0; }
};
std::mutex Fake::m;
std::map<void*, size_t> Fake::blocks;
size_t Fake::used = 0, Fake::limit = ~size_t(0) / 2;
int Fake::dev = 0, Fake::last_error = 0, Fake::frees = 0;
bool Fake::refuse = false, Fake::broken = false;
thread_local bool Fake::relaxed = false;
uintptr_t Fake::next = 4096;

typedef dcpse::DevicePoolT<Fake> Pool;

int main() {
    {
        Pool pool;
        void *a, *b, *c;
        CHECK(pool.alloc(&a, 5000) == 0);
        pool.free(a);
        CHECK(Fake::frees == 0);
        // the same block, after one wait
        CHECK(pool.alloc(&b, 4900) == 0 && b == a && Fake::frees == 1);
        // released before a known wait: no further one
        pool.free(b);
        CHECK(pool.wait() == 0 && Fake::frees == 2);
        CHECK(pool.alloc(&c, 5000) == 0 && c == a && Fake::frees == 2);
        // another device has its own waits and blocks
        pool.free(c);
        CHECK(pool.wait() == 0);
        Fake::dev = 1;
        CHECK(pool.alloc(&b, 5000) == 0 && b != a);
        Fake::dev = 0;
        pool.free(b);
        // a request that cannot be met gives the free blocks back
        CHECK(pool.alloc(&b, 100000) == 0);
        pool.free(b);
        Fake::limit = Fake::used + 50000;
        CHECK(pool.alloc(&c, 140000) == 0 && Fake::blocks.size() == 1 && Fake::last_error == 0);
        CHECK(pool.alloc(&b, 140000) == Fake::no_memory && b == nullptr);
        Fake::clear_error();
        Fake::limit = ~size_t(0) / 2;
        // no wait to be had: no block that may be in use is handed out, and no
        // error stays behind for the next launch to find
        pool.free(c);
        Fake::broken = true;
        CHECK(pool.wait() != 0 && Fake::last_error == 0);
        CHECK(pool.alloc(&a, 140000) != 0 && a == nullptr);
        Fake::broken = false;
        // under a capture the wait passes, a new allocation is refused as it was
        CHECK(pool.alloc(&c, 5000) == 0);
        pool.free(c);
        Fake::refuse = true;
        CHECK(pool.alloc(&a, 5000) == 0 && a == c);
        CHECK(pool.alloc(&b, 700000) != 0 && b == nullptr);
        pool.free(a);
        pool.release();
        CHECK(Fake::blocks.empty());
        Fake::refuse = false;
        Fake::clear_error();
        // sizes that no device has are refused (and end: doubling a unit up to
        // them would wrap around)
        Fake::limit = size_t(1) << 40;
        for (size_t absurd : {size_t(1) << 62, size_t(1) << 63, ~size_t(0) - 7, ~size_t(0)})
            CHECK(pool.alloc(&a, absurd) == Fake::no_memory && a == nullptr);
        Fake::clear_error();
        Fake::limit = ~size_t(0) / 2;
        // the last plan's end gives everything back
        CHECK(pool.alloc(&a, 3000) == 0);
        pool.free(a);
        pool.plan_created();
        pool.plan_created();
        pool.plan_destroyed();
        CHECK(!Fake::blocks.empty());
        pool.plan_destroyed();
        CHECK(Fake::blocks.empty() && Fake::used == 0);
        // no more than kPoolBytes are kept
        for (int i = 0; i < 6; ++i) CHECK(pool.alloc(&a, size_t(1) << 30) == 0 && (pool.free(a), true));
        std::set<void*> big;
        for (int i = 0; i < 6; ++i) {
            CHECK(pool.alloc(&a, size_t(1) << 30) == 0);
            big.insert(a);
        }
        for (void* p : big) pool.free(p);
        CHECK(Fake::used <= Pool::kPoolBytes);
        pool.release();
        CHECK(Fake::used == 0);
    }
    {
        // short of memory: a second try after something was given up, then less
        Pool pool;
        void *big, *p;
        Fake::limit = Fake::used + (size_t(1) << 20);
        CHECK(pool.alloc(&big, 900000) == 0);
        auto room = [&] {
            const bool had = big != nullptr;
            pool.free(big);
            big = nullptr;
            return had;
        };
        auto want = [&] { return pool.alloc(&p, 600000); };
        CHECK(dcpse::with_room<Fake>(want, room) == 0 && !big && p && Fake::last_error == 0);
        pool.free(p);
        Fake::limit = Fake::used;  // (the free block of 600,000 alone)
        auto more = [&] { return pool.alloc(&p, 2000000); };
        CHECK(dcpse::with_room<Fake>(more, room) == Fake::no_memory && !p);
        Fake::clear_error();
        Fake::limit = Fake::used + (size_t(1) << 20);
        for (long least : {1L, 100L, 3000L}) {
            long count = 4096;
            const int e = dcpse::with_less<Fake>(count, least, [&](long c) { return pool.alloc(&p, (size_t)c * 4000); });
            if (least == 3000) {
                CHECK(e == Fake::no_memory && count == 3000);
                Fake::clear_error();
            } else {
                CHECK(e == 0 && count == 256 && Fake::last_error == 0);
                pool.free(p);
            }
        }
        pool.release();
        Fake::limit = ~size_t(0) / 2;
    }
    {
        // what a captured call has read is not given up for room
        Pool pool;
        void *extra, *p;
        dcpse::KeptForGraphs kept;
        auto room = [&] {
            const bool had = extra && kept.may_go();
            if (had) pool.free(extra);
            if (had) extra = nullptr;
            return had;
        };
        auto want = [&] { return pool.alloc(&p, 900000); };
        for (bool captured : {true, false}) {
            Fake::limit = Fake::used + (size_t(1) << 20);
            CHECK(pool.alloc(&extra, 500000) == 0);
            kept = {};
            kept.used(false);
            kept.used(captured);
            kept.used(false);
            CHECK(dcpse::with_room<Fake>(want, room) == (captured ? Fake::no_memory : 0));
            CHECK((extra != nullptr) == captured);
            Fake::clear_error();
            pool.free(captured ? extra : p);
            pool.release();
        }
        Fake::limit = ~size_t(0) / 2;
    }
    {
        // threads: no two owners of a block at a time
        Pool pool;
        std::mutex m;
        std::set<void*> owned;
        bool bad = false;
        auto work = [&](unsigned seed) {
            std::mt19937 rng(seed);
            std::vector<void*> mine;
            for (int i = 0; i < 20000; ++i) {
                if (mine.size() < 8 && (rng() & 1)) {
                    void* p;
                    if (pool.alloc(&p, 512 << (rng() % 6)) != 0) bad = true;
                    std::lock_guard<std::mutex> lock(m);
                    if (!owned.insert(p).second) bad = true;
                    mine.push_back(p);
                } else if (!mine.empty()) {
                    void* p = mine.back();
                    mine.pop_back();
                    {
                        std::lock_guard<std::mutex> lock(m);
                        owned.erase(p);
                    }
                    pool.free(p);
                }
            }
            for (void* p : mine) {
                {
                    std::lock_guard<std::mutex> lock(m);
                    owned.erase(p);
                }
                pool.free(p);
            }
        };
        std::thread t[4] = {std::thread(work, 1), std::thread(work, 2), std::thread(work, 3), std::thread(work, 4)};
        for (auto& x : t) x.join();
        CHECK(!bad);
        pool.release();
        CHECK(Fake::used == 0);
    }
    return 0;
}
