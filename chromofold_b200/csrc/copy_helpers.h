// copy_helpers.h — threads that share a large checked copy of host rows (host_rows.h) with the thread that asks for it.
//
// With one thread copying, a prompt's rows reach the GPU at about 10 GB/s, a fifth of what the bus takes; with three helpers at 22 (2000
// rows to 8 heads, 16 MB: 1630 to 1700 us and 660 to 760 with all copies and launches; 1000 tokens with their attention, 1100 to 1200
// and 875 to 905). The first prompt of an adapter starts the threads and allocates the pinned memory. The copy is
// cut into pieces of 16 KB, which caller and helpers claim one by one: the caller never waits for a helper that has not claimed
// any, so that helpers which are asleep, or were never started, only leave it more to do.
// The helpers belong to one object, start with its first copy of kLeastFloats or more and end with it. After a copy they look for
// the next for kAwake and then sleep. One copy at a time: the owner is called by one thread at a time.
// A process that was forked has the object, but not its helpers: there the caller copies alone, and what they share is left as it
// is, for a helper may have held the lock or slept on the condition when the process was forked.
#ifndef CHROMOFOLD_B200_COPY_HELPERS_H
#define CHROMOFOLD_B200_COPY_HELPERS_H

#include <unistd.h>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <exception>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include "host_rows.h"

namespace cfb {

class CopyHelpers {
public:
    // Fewer are copied as fast by the caller alone, which has no one to wake. Appends of n rows of 128 floats to 8 heads, 3 ms (0.2 ms)
    // apart, alone and with helpers from four pieces on: 128 rows 252 and 255 us (250, 260), 160 rows 284 and 293 (276, 287), 192 rows
    // 316 and 315 (305, 304), 224 rows 357 and 326 (335, 322), 512 rows 509 and 313 (464, 303).
    static constexpr size_t kPieceFloats = 4096, kLeastFloats = 6 * kPieceFloats;
    static constexpr unsigned kHelpers = 3;   // four copies at once come near what the bus takes
    static constexpr std::chrono::microseconds kAwake{50};

    CopyHelpers() = default;
    CopyHelpers(const CopyHelpers &) = delete;
    CopyHelpers &operator=(const CopyHelpers &) = delete;
    ~CopyHelpers() {
        if (team_ && owner_ != getpid()) static_cast<void>(team_.release());
    }

    // chromofold_copy_max_magnitude, by several threads where that is worth it.
    uint32_t copy(float *dst, const float *src, size_t n) {
        if (n < kLeastFloats) return chromofold_copy_max_magnitude(dst, src, n);
        if (!team_) {
            owner_ = getpid();
            team_.reset(new (std::nothrow) Team);
        }
        if (!team_ || owner_ != getpid()) return chromofold_copy_max_magnitude(dst, src, n);
        return team_->copy(dst, src, n);
    }
    uint32_t asleep() const { return team_ ? team_->asleep() : 0u; }   // helpers that sleep

private:
    class Team {
    public:
        Team() {
            const unsigned processors = std::thread::hardware_concurrency();
            try {
                while (threads_.size() < kHelpers && threads_.size() + 1u < processors) threads_.emplace_back(&Team::help, this);
            } catch (const std::exception &) {   // no more threads, or no memory, to be had: those there are will do
            }
        }
        ~Team() {
            {
                std::lock_guard<std::mutex> hold(lock_);
                stop_ = true;
            }
            wake_.notify_all();
            for (std::thread &t : threads_) t.join();
        }
        uint32_t copy(float *dst, const float *src, size_t n) {
            dst_ = dst, src_ = src, n_ = n;
            const uint32_t pieces = static_cast<uint32_t>((n + kPieceFloats - 1) / kPieceFloats);
            top_.store(0, std::memory_order_relaxed);
            finished_.store(0, std::memory_order_relaxed);
            left_.store(++generation_ << 32 | pieces);   // from here on pieces can be claimed
            if (asleep_.load() != 0) {
                { std::lock_guard<std::mutex> hold(lock_); }   // who is about to sleep has seen the pieces, or is told
                wake_.notify_all();
            }
            while (work()) {}
            for (unsigned turn = 0; finished_.load(std::memory_order_acquire) != pieces; ++turn) pause(turn);
            return top_.load(std::memory_order_relaxed);
        }
        uint32_t asleep() const { return asleep_.load(); }

    private:
        // Claims a piece and copies it; false if none is left. A claim holds the copy open (finished_), so that what it reads of it stays.
        bool work() {
            uint64_t left = left_.load(std::memory_order_acquire);
            do {
                if (static_cast<uint32_t>(left) == 0u) return false;
            } while (!left_.compare_exchange_weak(left, left - 1u, std::memory_order_acq_rel, std::memory_order_acquire));
            const size_t begin = (static_cast<uint32_t>(left) - 1u) * kPieceFloats, count = n_ - begin < kPieceFloats ? n_ - begin : kPieceFloats;
            const uint32_t mine = chromofold_copy_max_magnitude(dst_ + begin, src_ + begin, count);
            for (uint32_t top = top_.load(std::memory_order_relaxed); top < mine && !top_.compare_exchange_weak(top, mine, std::memory_order_relaxed);) {}
            finished_.fetch_add(1u, std::memory_order_release);
            return true;
        }
        void help() {
            for (;;) {
                auto until = std::chrono::steady_clock::now() + kAwake;
                do {
                    if (work()) {
                        while (work()) {}
                        until = std::chrono::steady_clock::now() + kAwake;
                    }
                    for (unsigned turn = 0; turn < 64u && static_cast<uint32_t>(left_.load(std::memory_order_relaxed)) == 0u; ++turn) pause(0);
                } while (!stop_.load(std::memory_order_relaxed) && std::chrono::steady_clock::now() < until);
                std::unique_lock<std::mutex> hold(lock_);
                asleep_.fetch_add(1u);
                wake_.wait(hold, [&] { return stop_.load(std::memory_order_relaxed) || static_cast<uint32_t>(left_.load()) != 0u; });
                asleep_.fetch_sub(1u);
                if (stop_) return;
            }
        }
        static void pause(unsigned turn) {
            if (turn > 4096u) std::this_thread::yield();
#if defined(__x86_64__) || defined(__i386__)
            else __builtin_ia32_pause();
#endif
        }

        std::mutex lock_;
        std::condition_variable wake_;
        std::atomic<bool> stop_{false};
        std::atomic<uint32_t> asleep_{0}, finished_{0}, top_{0};
        std::atomic<uint64_t> left_{0};   // number of the copy << 32 | its pieces that nobody has claimed
        uint64_t generation_ = 0;
        float *dst_ = nullptr;
        const float *src_ = nullptr;
        size_t n_ = 0;
        std::vector<std::thread> threads_;
    };

    std::unique_ptr<Team> team_;
    pid_t owner_ = 0;   // the process that started them
};

}  // namespace cfb

#endif
