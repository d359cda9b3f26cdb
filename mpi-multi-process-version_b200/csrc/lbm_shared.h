// Host-side bookkeeping that handles on several devices and threads share.
#ifndef LBM_SHARED_H
#define LBM_SHARED_H
#include <stdint.h>

#include <atomic>

namespace lbm {

// A set-up call that holds for one device only (cudaFuncSetAttribute): made once
// for each device, and again as long as it fails.
class OncePerDevice {
    std::atomic<uint64_t> done_{0};

public:
    template <class F>
    auto run(int device, F call) -> decltype(call())
    {
        using E = decltype(call());
        const uint64_t bit = device >= 0 && device < 64 ? uint64_t(1) << device : 0;
        if (done_.load(std::memory_order_acquire) & bit) return E(0);
        const E e = call();
        if (e == E(0)) done_.fetch_or(bit, std::memory_order_release);
        return e;
    }
};

// Kernels launched, by all threads.  A thread that captures a graph takes its own
// launches since a mark out of the count again: they count when the graph is
// replayed, and other threads' launches in the meantime count as ever.
class LaunchCount {
    std::atomic<int64_t> total_{0};
    static int64_t &mine()
    {
        static thread_local int64_t n = 0;
        return n;
    }

public:
    void operator+=(int64_t n)
    {
        total_.fetch_add(n, std::memory_order_relaxed);
        mine() += n;
    }
    void operator++() { *this += 1; }
    int64_t total() const { return total_.load(std::memory_order_relaxed); }
    int64_t mark() const { return mine(); }
    int64_t take(int64_t mark)
    {
        const int64_t n = mine() - mark;
        *this += -n;
        return n;
    }
};

}  // namespace lbm
#endif
