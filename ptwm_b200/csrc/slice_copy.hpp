// Moves bytes that arrive slice by slice in a ring of staging slots on to where they belong, with a few host threads.  Standard
// library only: what fills the slots is the caller's.
#pragma once
#include <algorithm>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace ptwm {

enum class Moved { all, failed, no_threads };

struct StartThread {
    template <class F>
    std::thread operator()(F&& f) const { return std::thread(std::forward<F>(f)); }
};

// Slice k (of `slice` bytes, the last one what is left of `n`) passes through slot k mod `ring` of `stage`.  `send(k)` begins to
// fill the slot and `arrived(k)` waits until it is full; both return false on an error and throw nothing.  Up to `n_threads`
// threads move slices; it does with as many as can be started, and when none can nothing has been sent yet.  After `failed`
// slots may still be being filled.  No thread outlives the call.
template <class Send, class Arrived, class Start = StartThread>
Moved move_slices(uint8_t* dst, const uint8_t* stage, size_t n, size_t slice, size_t ring, size_t n_threads, Send&& send, Arrived&& arrived, Start&& start = Start{}) {
    const size_t slices = (n + slice - 1) / slice;
    std::mutex mu;
    std::condition_variable cv;
    size_t sent = 0, next = 0;           // slices sent; the next one a thread takes on
    std::vector<char> moved(slices, 0);  // slices that have left their slot
    bool failed = false;
    auto work = [&]() {
        for (;;) {
            size_t k;
            {
                std::unique_lock<std::mutex> l(mu);
                k = next;
                if (k >= slices) return;
                ++next;
                cv.wait(l, [&] { return sent > k || failed; });
                if (failed) return;
            }
            const bool ok = arrived(k);
            if (ok) std::memcpy(dst + k * slice, stage + (k % ring) * slice, std::min(slice, n - k * slice));
            std::lock_guard<std::mutex> l(mu);
            if (!ok) failed = true;
            moved[k] = 1;
            cv.notify_all();
        }
    };
    std::vector<std::thread> threads;
    threads.reserve(n_threads);
    struct Join {  // whatever ends the call, the threads are told and waited for
        std::vector<std::thread>& threads;
        std::mutex& mu;
        std::condition_variable& cv;
        bool &failed, done = false;
        ~Join() {
            if (!done) { { std::lock_guard<std::mutex> l(mu); failed = true; } cv.notify_all(); }
            for (auto& t : threads) t.join();
        }
    };
    {
        Join join{threads, mu, cv, failed};
        for (size_t t = 0; t < std::min(n_threads, slices); ++t) {
            try { threads.push_back(start(work)); }
            catch (const std::system_error&) { break; }
        }
        if (threads.empty()) return Moved::no_threads;
        for (size_t k = 0; k < slices; ++k) {
            std::unique_lock<std::mutex> l(mu);
            if (k >= ring) cv.wait(l, [&] { return moved[k - ring] || failed; });
            if (failed) break;
            l.unlock();
            const bool ok = send(k);
            l.lock();
            if (ok) sent = k + 1; else failed = true;
            cv.notify_all();
            if (!ok) break;
        }
        join.done = true;  // every slice was sent, or `failed` says otherwise
    }
    return failed ? Moved::failed : Moved::all;
}

}  // namespace ptwm
