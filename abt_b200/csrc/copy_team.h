// copy_pool.h -- helper threads for the host side of large copies.
//
// A context's large copies move each chunk between the caller's array and a pinned slot
// while the next chunk is in transfer (ctx.cu).  One thread moves 10 to 14 GB/s, the link
// 50 and more, so helpers take pieces of a chunk beside the caller.
//
// * Pieces are claimed one at a time, and the caller moves what nobody has claimed, so a
//   helper that does not run takes nothing.  One that is taken off its core within a piece is
//   waited for, a slice of the scheduler's (4 ms).  So after a wait of kStallUs the next copies
//   go without helpers, kRest of them and twice as many after each further one.
// * Helpers look for the next chunk, or the next copy, for kSpinUs and then sleep.
// * No more threads than the caller may use: the processors it is bound to and OpenMP's
//   limit (OMP_NUM_THREADS) count, copies under way at once share the processors, and
//   inside a parallel region the caller works alone.
//
// Measured on 16 cores, a call that returns 2.1 MB, against an OpenMP team of eight with a
// barrier a chunk (whose threads also spin for milliseconds after a copy) and the driver's copy:
// idle host 120 us (117, 185); every core busy, mean 0.27 to 0.38 ms (0.3 to 3.8, 0.34 to 0.41);
// bound to one core 195 us (317, 183); 16 threads with a context each 58 us a call (58, 210).
// Two such grids a call on a busy host: mean 1.4 to 1.5 ms (1.3 to 64, 1.3 to 1.4).
#pragma once
#include <omp.h>
#include <sched.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace pbt {

class CopyPool {
public:
    static constexpr int kMaxHelpers = 7;
    static constexpr size_t kPiece = (size_t)64 << 10;
    static constexpr int kSpinUs = 100, kStallUs = 1000, kRest = 256, kMostRest = 16384;
    using Move = void (*)(char *, const char *, size_t);

    explicit CopyPool(Move move = [](char *d, const char *s, size_t n) { memcpy(d, s, n); }) : move_(move) {}

    // Helpers that the calling thread may use now, one of `copies` under way in the process.
    static int allowed(int copies = 1) {
        if (omp_in_parallel()) return 0;
        cpu_set_t set;
        const int cpus = sched_getaffinity(0, sizeof set, &set) == 0 ? CPU_COUNT(&set)
                                                                      : (int)std::thread::hardware_concurrency();
        return std::max(0, std::min({cpus / std::max(copies, 1), omp_get_max_threads(), kMaxHelpers + 1}) - 1);
    }

    ~CopyPool() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            quit_ = true;
        }
        cv_.notify_all();
        for (std::thread &t : threads_) t.join();
    }

    // Calls the helpers to a copy of one or more chunks.  Helpers that cannot be started
    // are done without.
    void begin() {
        helped_ = false;
        const int copies = ++copying();
        if (skip_ > 0) {
            skip_--;
            return;
        }
        const int want = allowed(copies);
        try {
            threads_.reserve(kMaxHelpers);
            while ((int)threads_.size() < want) {
                const int i = (int)threads_.size();
                threads_.emplace_back([this, i] { helper(i); });
            }
        } catch (const std::exception &) {
        }
        const int n = std::min(want, (int)threads_.size());
        if (!n) return;
        helped_ = true;
        active_.store(n, std::memory_order_relaxed);
        wake();
    }

    // One chunk; returns when all of it is in dst.
    void run(char *dst, const char *src, size_t n) {
        if (!n) return;
        if (!helped_) {
            move_(dst, src, n);
            return;
        }
        if (asleep_.load(std::memory_order_relaxed) > 0) wake();  // the first chunk took long to come
        // one word holds the chunk's number, its pieces and the next piece to claim, so
        // that a late claim of an earlier chunk can never succeed
        piece_ = std::max(kPiece, ((n + 0xfffe) / 0xffff + 63) & ~(size_t)63);
        const uint64_t np = (n + piece_ - 1) / piece_;
        dst_ = dst;
        src_ = src;
        n_ = n;
        done_.store(0, std::memory_order_relaxed);
        word_.store(++chunk_ << 32 | np << 16, std::memory_order_release);
        while (piece()) {
        }
        if (done_.load(std::memory_order_acquire) == np) return;
        const auto t0 = Clock::now();
        while (done_.load(std::memory_order_acquire) < np) {
            if (past(t0, kStallUs))
                std::this_thread::sleep_for(std::chrono::microseconds(50));
            else
                __builtin_ia32_pause();
        }
        if (past(t0, kStallUs)) {
            skip_ = rest_;
            rest_ = std::min(2 * rest_, kMostRest);
            smooth_ = 0;
            helped_ = false;  // the rest of this copy alone too
        }
    }

    void end() {
        if (helped_ && ++smooth_ == kRest) rest_ = kRest;
        helped_ = false;
        --copying();
    }

private:
    // Copies under way in the process, which share its processors.
    static std::atomic<int> &copying() {
        static std::atomic<int> n{0};
        return n;
    }

    void wake() {
        bool any;
        {
            std::lock_guard<std::mutex> lk(mu_);
            epoch_++;
            any = asleep_.load(std::memory_order_relaxed) > 0;
        }
        if (any) cv_.notify_all();
    }

    // Claims and moves a piece of the current chunk; false: none is left.
    bool piece() {
        uint64_t w = word_.load(std::memory_order_acquire);
        do {
            if ((w & 0xffff) >= (w >> 16 & 0xffff)) return false;
        } while (!word_.compare_exchange_weak(w, w + 1, std::memory_order_acq_rel, std::memory_order_acquire));
        // the chunk's fields stay until this piece is counted
        const size_t o = (w & 0xffff) * piece_;
        move_(dst_ + o, src_ + o, std::min(piece_, n_ - o));
        done_.fetch_add(1, std::memory_order_release);
        return true;
    }

    using Clock = std::chrono::steady_clock;
    static bool past(Clock::time_point t0, int us) { return Clock::now() - t0 > std::chrono::microseconds(us); }

    void helper(int i) {
        uint64_t seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> lk(mu_);
                asleep_++;
                cv_.wait(lk, [&] { return quit_ || (epoch_ != seen && active_.load(std::memory_order_relaxed) > i); });
                asleep_--;
                if (quit_) return;
                seen = epoch_;
            }
            Clock::time_point last = Clock::now();
            for (int idle = 0; active_.load(std::memory_order_relaxed) > i;) {
                if (piece()) {
                    idle = 0;
                    continue;
                }
                if (idle++ == 0) last = Clock::now();
                __builtin_ia32_pause();
                if (idle % 64 == 0 && past(last, kSpinUs)) break;
            }
        }
    }

    const Move move_;
    std::vector<std::thread> threads_;
    std::mutex mu_;
    std::condition_variable cv_;
    uint64_t epoch_ = 0;  // calls of the helpers
    std::atomic<int> asleep_{0};
    bool quit_ = false;
    std::atomic<int> active_{0};  // helpers that the latest copy may use
    bool helped_ = false;
    int skip_ = 0, rest_ = kRest, smooth_ = 0;  // copies to go without; the next such rest; copies since the last stall
    uint64_t chunk_ = 0;
    char *dst_ = nullptr;
    const char *src_ = nullptr;
    size_t n_ = 0, piece_ = kPiece;
    alignas(64) std::atomic<uint64_t> word_{0};
    alignas(64) std::atomic<uint64_t> done_{0};
};

}  // namespace pbt
