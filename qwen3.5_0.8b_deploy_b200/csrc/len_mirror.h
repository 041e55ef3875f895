// When the host's mirror of lengths that live on the device may be behind them, and when it is known not to be.
#pragma once

#include <atomic>
#include <cstdint>
#include <mutex>

namespace b200 {

// Every launch that advances the lengths without the host marks the mirror.  Marks are counted, in all and by the thread that makes them: whoever brings the
// mirror up to date answers for the marks that it knows of, and a step that another thread launches meanwhile keeps its own.
class MirrorMarks {
public:
    struct Point { uint64_t all, own; };
    void mark() {
        ++own();
        all_.fetch_add(1);
    }
    bool behind() const { return seen_.load() != all_.load(); }
    Point here() const { return {all_.load(), own()}; }

    // `read` waits for the device and takes the lengths over (0, or an error to pass on).
    template <typename F>
    int refresh(F&& read) {
        if (!behind()) return 0;
        std::lock_guard<std::mutex> hold(lock_);
        const uint64_t at = all_.load();
        if (seen_.load() == at) return 0;
        const int status = read();
        if (status == 0) seen_.store(at);
        return status;
    }
    // The mirror was up to date at `at`, and the steps that this thread launched since are over: `enter` adds what they did.  Left to the next refresh
    // when anyone else marked the mirror meanwhile, or read it.
    template <typename F>
    void enter_own(Point at, F&& enter) {
        std::lock_guard<std::mutex> hold(lock_);
        const uint64_t now = at.all + (own() - at.own);
        if (seen_.load() != at.all || all_.load() != now) return;
        enter();
        seen_.store(now);
    }
    // The lengths were set on both sides.
    template <typename F>
    void set_both(F&& set) {
        std::lock_guard<std::mutex> hold(lock_);
        set();
        seen_.store(all_.load());
    }

private:
    static uint64_t& own() {
        static thread_local uint64_t n = 0;
        return n;
    }
    std::atomic<uint64_t> all_{0}, seen_{0};
    std::mutex lock_;
};

}  // namespace b200
