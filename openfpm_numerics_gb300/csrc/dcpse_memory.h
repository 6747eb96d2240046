// dcpse_memory.h -- device memory of the plans.
//
// A freed block is kept for the next request of about its size instead of going
// back to the driver, whose cudaMalloc and cudaFree cost 10 us to 1 ms each for
// blocks of a megabyte and more (a neighbour build makes 14 of each, an operator
// update of 4,096 particles spent 0.6 of its 1.0 ms there).  Shared by all plans
// and threads of the process, since an operator update builds its list on a plan
// of its own.  Bounded: at most kPoolBytes of free blocks per process, given back
// when a request cannot be met and when the last plan is destroyed.
//
// cudaFree waits for the device.  Here a block is handed out again only after
// such a wait that came later than its release (wait()), so whatever stream or
// thread still used it when it was freed has finished.  The wait is a cudaFree
// itself, of a block of one byte: 2.2 us on an idle GPU with its cudaMalloc.  A
// cudaDeviceSynchronize (0.6 us) is invalid while any stream of the device is
// captured and ends that capture, also one of another thread in thread-local
// mode, where cudaMalloc and cudaFree are allowed.  Inside the wait and a release
// they are allowed in captures of any mode, this thread's too: a plan that is
// destroyed meanwhile (by a garbage collector, say) does not end them.
//
// Rt: the runtime's calls (CudaRt, or a fake in the host tests).
#pragma once

#include <algorithm>
#include <cstddef>
#include <map>
#include <mutex>
#include <unordered_map>
#include <utility>

namespace dcpse {

template <class Rt>
class DevicePoolT {
public:
    typedef typename Rt::Error Error;
    static constexpr size_t kPoolBytes = size_t(4) << 30;

    Error alloc(void** p, size_t want) {
        *p = nullptr;
        int dev = 0;
        Error e = Rt::device(&dev);
        if (e != Rt::ok) return e;
        size_t bytes = rounded(want);
        bool waiting = false;  // a block would do once it is known to be idle
        {
            std::lock_guard<std::mutex> lock(m_);
            if (take(p, dev, bytes)) return Rt::ok;
            waiting = find(dev, bytes, ~0ull) != free_.end();
        }
        if (waiting && wait() == Rt::ok) {
            std::lock_guard<std::mutex> lock(m_);
            if (take(p, dev, bytes)) return Rt::ok;
        }
        e = Rt::malloc(p, bytes);
        if (e == Rt::no_memory) {
            Rt::clear_error();
            release();
            bytes = want;
            e = Rt::malloc(p, bytes);
        }
        if (e == Rt::ok) {
            // (a block that cannot be noted goes back to the driver when freed)
            noted([&] { live_[*p] = Block{bytes, dev, 0}; });
        } else {
            *p = nullptr;
        }
        return e;
    }
    void free(void* p) {
        if (!p) return;
        bool kept = false;
        noted([&] {
            auto it = live_.find(p);
            if (it == live_.end()) return;
            Block b = it->second;
            live_.erase(it);
            if (cached_ + b.bytes > kPoolBytes) return;
            b.stamp = ++stamp_;
            free_.emplace(b.bytes, std::make_pair(p, b));
            cached_ += b.bytes;
            kept = true;
        });
        if (!kept) Rt::free(p);
    }
    // What cudaFree does beside freeing: returns when the work that was submitted
    // to the current device, on any stream, is done.
    Error wait() {
        int dev = 0;
        Error e = Rt::device(&dev);
        if (e != Rt::ok) return e;
        unsigned long long stamp;
        {
            std::lock_guard<std::mutex> lock(m_);
            stamp = stamp_;
        }
        {
            typename Rt::Relaxed relaxed;
            void* p = nullptr;
            e = Rt::malloc(&p, 1);
            if (e == Rt::ok) e = Rt::free(p);
        }
        if (e == Rt::ok)
            noted([&] { synced_[dev] = std::max(synced_[dev], stamp); });
        else
            Rt::clear_error();
        return e;
    }
    void plan_created() {
        std::lock_guard<std::mutex> lock(m_);
        ++plans_;
    }
    void plan_destroyed() {
        bool last;
        {
            std::lock_guard<std::mutex> lock(m_);
            last = --plans_ == 0;
        }
        if (last) release();
    }
    // every free block back to the driver
    void release() {
        FreeMap blocks;
        {
            std::lock_guard<std::mutex> lock(m_);
            blocks.swap(free_);
            cached_ = 0;
        }
        typename Rt::Relaxed relaxed;
        for (auto& f : blocks) Rt::free(f.second.first);  // (any device's: pointers are unified)
    }

private:
    struct Block {
        size_t bytes;
        int dev;
        unsigned long long stamp;  // order of the releases
    };
    using FreeMap = std::multimap<size_t, std::pair<void*, Block>>;
    // fn under the lock; its bookkeeping may fail for want of host memory, which
    // must not leave a C entry point as an exception
    template <class Fn>
    void noted(Fn fn) {
        std::lock_guard<std::mutex> lock(m_);
        try {
            fn();
        } catch (...) {
        }
    }
    // sixteenths of a power of two, at least 512 bytes: lists and weights of
    // moving particles change a little in size from step to step (sizes that no
    // device has are left as they are, for the driver to refuse)
    static size_t rounded(size_t want) {
        if (want >= size_t(1) << 48) return want;
        size_t unit = 512;
        while (unit * 32 <= want) unit *= 2;
        return (want + unit - 1) / unit * unit;
    }
    // a free block of this device of `bytes` or up to an eighth more, released
    // before the device's last known wait
    typename FreeMap::iterator find(int dev, size_t bytes, unsigned long long synced) {
        for (auto it = free_.lower_bound(bytes); it != free_.end() && it->first <= bytes + bytes / 8; ++it)
            if (it->second.second.dev == dev && it->second.second.stamp <= synced) return it;
        return free_.end();
    }
    bool take(void** p, int dev, size_t bytes) {
        auto known = synced_.find(dev);
        auto it = find(dev, bytes, known == synced_.end() ? 0ull : known->second);
        if (it == free_.end()) return false;
        try {
            live_[it->second.first] = it->second.second;
        } catch (...) {
            return false;
        }
        *p = it->second.first;
        cached_ -= it->first;
        free_.erase(it);
        return true;
    }
    std::mutex m_;
    std::unordered_map<void*, Block> live_;
    FreeMap free_;
    std::unordered_map<int, unsigned long long> synced_;
    unsigned long long stamp_ = 0;
    size_t cached_ = 0;
    int plans_ = 0;
};

// alloc(), and where memory is short once more after room() has given something up
// (it returns whether it had anything)
template <class Rt, class Alloc, class Room>
typename Rt::Error with_room(Alloc alloc, Room room) {
    typename Rt::Error e = alloc();
    if (e == Rt::no_memory && room()) {
        Rt::clear_error();
        e = alloc();
    }
    return e;
}

// alloc(count), with count halved (down to `least`) while memory is short
template <class Rt, class Int, class Alloc>
typename Rt::Error with_less(Int& count, Int least, Alloc alloc) {
    for (;;) {
        const typename Rt::Error e = alloc(count);
        if (e != Rt::no_memory || count <= least) return e;
        Rt::clear_error();
        count = std::max(least, count / 2);
    }
}

// Whether an optional buffer may be given up for room: not once a call that was
// captured has read it, since the graph keeps its address and may run at any time
// while the plan's layout lives.
class KeptForGraphs {
public:
    void used(bool capturing) { kept_ = kept_ || capturing; }
    bool may_go() const { return !kept_; }

private:
    bool kept_ = false;
};

}  // namespace dcpse
