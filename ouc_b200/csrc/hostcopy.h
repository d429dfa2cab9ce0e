// Host side of large copies from the device (hostio.cu), apart from the CUDA
// calls so that it also runs without a GPU.
#pragma once
#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstring>
#include <functional>
#include <system_error>
#include <thread>
#include <vector>

namespace ouc {
namespace host {

struct HostCopy {
    void* host;
    void* dev;
    size_t bytes;
};

// Whether two of the arrays share bytes: their copies must then be made in order.
inline bool overlapping(std::vector<HostCopy> c) {
    c.erase(std::remove_if(c.begin(), c.end(), [](const HostCopy& x) { return x.bytes == 0; }), c.end());
    std::sort(c.begin(), c.end(), [](const HostCopy& a, const HostCopy& b) { return std::less<void*>()(a.host, b.host); });
    for (size_t k = 1; k < c.size(); ++k)
        if (std::less<char*>()(static_cast<char*>(c[k].host), static_cast<char*>(c[k - 1].host) + c[k - 1].bytes)) return true;
    return false;
}

// Run `worker` on up to n new threads and `caller` on this one, then join
// them.  Where the system gives fewer threads, those that started do the work;
// with none at all `caller` is not run and the result is false.
template <class Worker, class Caller>
bool run_team(int n, Worker&& worker, Caller&& caller) {
    std::vector<std::thread> team;
    try {
        team.reserve(n);
        for (int t = 0; t < n; ++t) team.emplace_back(worker);
    } catch (const std::exception&) {   // no thread, or no memory for one
    }
    if (team.empty()) return false;
    caller();
    for (auto& t : team) t.join();
    return true;
}

// Bring `copies` to the host through a ring of `slots` buffers of `chunk`
// bytes: this thread queues chunk after chunk, queue(slot, device address,
// bytes), into slots that are free, and a team of `threads` takes the chunks
// in turn, waits for each, wait(slot), and moves it on to its array.  queue and
// wait return 0 or an error; the first error ends the copy.  Returns it, or
// -1 when no thread could be started (nothing has been queued then).
template <class Queue, class Wait>
int ring_copy(const std::vector<HostCopy>& copies, char* ring, size_t chunk, int slots, int threads, Queue&& queue,
              Wait&& wait) {
    std::vector<HostCopy> chunks;
    for (const auto& x : copies)
        for (size_t o = 0; o < x.bytes; o += chunk)
            chunks.push_back({static_cast<char*>(x.host) + o, static_cast<char*>(x.dev) + o,
                              x.bytes - o < chunk ? x.bytes - o : chunk});
    const int n = (int)chunks.size();
    // chunk k lives in slot k % slots.  moved[s] counts the chunks of slot s
    // that the team has moved on, queued the chunks whose copies into the ring
    // have been queued.
    std::vector<std::atomic<int>> moved(slots);
    std::atomic<int> queued{0}, next{0}, error{0};
    for (auto& m : moved) m = 0;
    auto failed = [&](int e) {
        int none = 0;
        if (e) error.compare_exchange_strong(none, e);
        return error.load() != 0;
    };
    auto worker = [&]() {
        for (int k; (k = next.fetch_add(1)) < n;) {
            const int s = k % slots;
            while (queued.load(std::memory_order_acquire) <= k && !failed(0)) std::this_thread::yield();
            if (failed(0) || failed(wait(s))) return;
            memcpy(chunks[k].host, ring + (size_t)s * chunk, chunks[k].bytes);
            moved[s].fetch_add(1, std::memory_order_release);
        }
    };
    const bool ran = run_team(threads < n ? threads : n, worker, [&]() {
        for (int k = 0; k < n; ++k) {
            const int s = k % slots;
            while (moved[s].load(std::memory_order_acquire) < k / slots && !failed(0)) std::this_thread::yield();
            if (failed(0) || failed(queue(s, chunks[k].dev, chunks[k].bytes))) return;
            queued.store(k + 1, std::memory_order_release);
        }
    });
    return ran || n == 0 ? error.load() : -1;
}

}  // namespace host
}  // namespace ouc
