/* Host threads for the copies and conversions of whole rasters. */
#ifndef SW2D_THREADS_H
#define SW2D_THREADS_H

#include <algorithm>
#include <cstddef>
#include <exception>
#include <thread>
#include <vector>

namespace sw2d {

/* f(first, last) over [0, n), split across at most nt threads.  What a thread
 * that cannot be started was to do, the caller does: the entry points are C,
 * so no exception may leave them. */
template <typename F>
void split_over_threads(size_t n, size_t nt, F f) {
    const size_t per = nt > 1 ? (n + nt - 1) / nt : n;
    size_t done = 0;
    std::vector<std::thread> th;
    try {
        if (per < n) th.reserve(nt);
        for (; per < n && done < n; done += per)
            th.emplace_back([f, done, last = std::min(n, done + per)] { f(done, last); });
    } catch (const std::exception&) { /* no thread or no memory for one */
    }
    if (done < n) f(done, n);
    for (auto& x : th) x.join();
}

} // namespace sw2d

#endif /* SW2D_THREADS_H */
