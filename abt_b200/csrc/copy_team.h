// copy_team.h -- several host threads for the host side of large copies.
//
// A context's large copies move each chunk between the caller's array and a pinned slot
// while the next chunk is in transfer (ctx.cu).  One thread moves 10 to 14 GB/s, the link
// 50 and more, so a chunk is shared out among an OpenMP team: the same threads as the
// library's other parallel loops, which wait actively between the chunks.  (Threads of
// their own would be taken for load beside a team of all cores that still spins, and two of
// its threads end up on one core: an FP64 diff_main of 2.3 ms took 5.4.)
//
// * No more threads than the caller may use: the processors it is bound to and OpenMP's
//   limit (OMP_NUM_THREADS) count, and inside a parallel region the caller works alone.
// * On a host whose cores are busy the team's barrier waits for the scheduler, slices of
//   4 ms and more.  After a wait of kStallUs the rest of the copy and the next kRest copies
//   are the caller's alone, and twice as many after each further such wait.
//
// Measured on 16 cores, a call that returns 2.1 MB (in brackets: a team of eight whatever the
// host, and the driver's copy): idle host 114 us (116, 185); bound to one core 193 us (317,
// 190); every core busy, means of 0.26 to 0.36 ms (0.3 to 9.4, 0.34 to 0.41).  Two such grids a
// call on a busy host: 1.3 to 1.4 ms (1.0 to 64, 1.3 to 1.4).
#pragma once
#include <omp.h>
#include <sched.h>
#include <string.h>

#include <algorithm>
#include <chrono>
#include <cstdint>

namespace pbt {

class CopyTeam {
public:
    static constexpr int kMost = 8;
    static constexpr size_t kPiece = (size_t)64 << 10;
    static constexpr int kStallUs = 2000, kRest = 256, kMostRest = 16384;
    using Move = void (*)(char *, const char *, size_t);

    explicit CopyTeam(Move move = [](char *d, const char *s, size_t n) { memcpy(d, s, n); }) : move_(move) {}

    // Threads that the caller may use now, itself among them.
    static int allowed() {
        if (omp_in_parallel()) return 1;
        cpu_set_t set;
        const int cpus = sched_getaffinity(0, sizeof set, &set) == 0 ? CPU_COUNT(&set) : omp_get_num_procs();
        return std::max(1, std::min({cpus, omp_get_max_threads(), kMost}));
    }

    // Around the chunks of a copy.
    void begin() {
        threads_ = skip_ > 0 ? 1 : allowed();
        if (skip_ > 0) skip_--;
    }
    void end() {
        if (threads_ > 1 && ++smooth_ == kRest) rest_ = kRest;
    }

    // One chunk; returns when all of it is in dst.
    void run(char *dst, const char *src, size_t n) {
        const int64_t np = (int64_t)((n + kPiece - 1) / kPiece);
        if (threads_ <= 1 || np <= 1) {
            if (n) move_(dst, src, n);
            return;
        }
        Clock::time_point done;  // the caller has found no further piece
#pragma omp parallel num_threads(threads_)
        {
#pragma omp for schedule(static) nowait
            for (int64_t i = 0; i < np; i++)
                move_(dst + i * kPiece, src + i * kPiece, std::min(kPiece, n - i * kPiece));
            if (omp_get_thread_num() == 0) done = Clock::now();
        }
        if (Clock::now() - done > std::chrono::microseconds(kStallUs)) {
            threads_ = 1;
            skip_ = rest_;
            rest_ = std::min(2 * rest_, kMostRest);
            smooth_ = 0;
        }
    }

private:
    using Clock = std::chrono::steady_clock;
    const Move move_;
    int threads_ = 1;                           // of the copy under way
    int skip_ = 0, rest_ = kRest, smooth_ = 0;  // copies to do alone; the next such rest; copies since the last stall
};

}  // namespace pbt
