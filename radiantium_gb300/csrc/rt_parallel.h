/*
 * rt_parallel.h - a loop over host threads, and the arrays it fills.
 */
#ifndef RT_PARALLEL_H
#define RT_PARALLEL_H

#include <stdint.h>
#include <algorithm>
#include <exception>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <utility>
#include <vector>

namespace rtb {

/* A vector whose new elements are not zeroed: resize() leaves the pages of a
 * large array untouched, so that the threads that fill it also fault it in. */
template <class T>
struct NoInit : std::allocator<T> {
    template <class U> struct rebind { typedef NoInit<U> other; };
    template <class U> void construct(U* p) { ::new ((void*)p) U; }
    template <class U, class... A> void construct(U* p, A&&... a) { ::new ((void*)p) U(std::forward<A>(a)...); }
};
template <class T> using Array = std::vector<T, NoInit<T>>;

/* f(begin, end) over [0, n), split into up to one range per host core of at
 * least `grain` elements each.  The first exception of a range is rethrown
 * here once every thread has ended; where no thread can be started the
 * ranges run here. */
template <class F>
void parallel_for(int64_t n, int64_t grain, F&& f) {
    if (n <= 0) return;
    static const int64_t cores = std::max(1u, std::thread::hardware_concurrency());   /* it reads /sys */
    const int64_t parts = std::min(cores, n / std::max<int64_t>(1, grain));
    if (parts <= 1) {
        f((int64_t)0, n);
        return;
    }
    std::exception_ptr failed;
    std::mutex lock;
    auto range = [&](int64_t k) {
        try {
            f(n * k / parts, n * (k + 1) / parts);
        } catch (...) {
            std::lock_guard<std::mutex> g(lock);
            if (!failed) failed = std::current_exception();
        }
    };
    std::vector<std::thread> threads;
    threads.reserve((size_t)parts);
    int64_t k = 1;
    try {
        for (; k < parts; k++) threads.emplace_back(range, k);
    } catch (...) {                            /* no thread, or no memory for its state: the rest runs here */
    }
    range(0);
    for (; k < parts; k++) range(k);
    for (std::thread& t : threads) t.join();
    if (failed) std::rethrow_exception(failed);
}

}  // namespace rtb

#endif
