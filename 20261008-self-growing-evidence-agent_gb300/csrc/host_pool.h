// host_pool.h -- a persistent pool of host threads for the miner's per-node
// bookkeeping between device waves.
//
// run(n, chunk, fn) calls fn(lo, hi) on chunks of [0, n) taken from a shared
// counter by the caller and the pool's threads, and returns when every chunk
// is done.  A thread that is still asleep is not waited for: a job is over when
// its chunks are (waiting for every thread to wake up and look took most of the
// time of the jobs after a device wave).  The threads start on first use.  Between calls they poll for the
// next job for a short while (a wave issues several jobs within a
// millisecond or two), then sleep on a condition variable.  One owner thread
// issues the jobs, one at a time: run() is not reentrant (fn must not call it)
// and a pool is not shared between threads (each miner owns its own).
#pragma once

#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <mutex>
#include <thread>
#include <type_traits>
#include <vector>

namespace sg {

class HostPool {
  public:
    explicit HostPool(unsigned threads) : n_(std::max(1u, threads)) {}
    HostPool(const HostPool &) = delete;
    HostPool &operator=(const HostPool &) = delete;
    ~HostPool() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            stop_.store(true, std::memory_order_relaxed);
        }
        cv_.notify_all();
        for (auto &t : th_) t.join();
    }

    unsigned threads() const { return n_; }

    // fn(lo, hi) over [0, n) in chunks of `chunk`; serial when n is at most one chunk
    template <class F> void run(uint64_t n, uint64_t chunk, F &&fn) {
        if (n == 0) return;
        chunk = std::max<uint64_t>(chunk, 1);
        if (n_ == 1 || n <= chunk) {
            fn((uint64_t)0, n);
            return;
        }
        if (th_.empty()) start();
        chunk = std::max(chunk, n / (kMaxChunks - 1) + 1);
        call_ = [](void *f, uint64_t lo, uint64_t hi) { (*static_cast<std::remove_reference_t<F> *>(f))(lo, hi); };
        fn_ = const_cast<void *>(static_cast<const void *>(&fn));
        n_job_ = n;
        chunk_ = chunk;
        const uint64_t n_chunks = (n + chunk - 1) / chunk;
        finished_.store(0, std::memory_order_relaxed);
        {
            std::lock_guard<std::mutex> lk(mu_);
            ticket_.store(n_chunks << kIdxBits, std::memory_order_release);
        }
        cv_.notify_all();
        work();
        auto done = [&] { return finished_.load(std::memory_order_acquire) == n_chunks; };
        if (!poll(done)) {
            std::unique_lock<std::mutex> lk(mu_);
            done_.wait(lk, done);
        }
    }

  private:
    // polls cond() for up to kPollUs microseconds
    template <class C> static bool poll(C &&cond) {
        constexpr int64_t kPollUs = 200;
        const auto t0 = std::chrono::steady_clock::now();
        for (uint32_t i = 0;; ++i) {
            if (cond()) return true;
            if ((i & 255) == 255 &&
                std::chrono::duration_cast<std::chrono::microseconds>(std::chrono::steady_clock::now() - t0).count() >
                    kPollUs)
                return cond();
        }
    }
    void start() {
        th_.reserve(n_ - 1);
        for (unsigned i = 1; i < n_; ++i) th_.emplace_back([this] { loop(); });
    }
    // A ticket holds the job's number of chunks and the next one to take, so that a late thread
    // sees from the ticket alone that nothing is left.  The job's other fields are read only with
    // a chunk in hand: they stay as they are until that chunk is reported finished.
    static bool open(uint64_t t) { return (t & kIdxMask) < (t >> kIdxBits); }
    void work() {
        while (open(ticket_.load(std::memory_order_relaxed))) {
            const uint64_t t = ticket_.fetch_add(1, std::memory_order_acq_rel);
            if (!open(t)) return;
            const uint64_t lo = (t & kIdxMask) * chunk_, n_chunks = t >> kIdxBits;
            call_(fn_, lo, std::min(n_job_, lo + chunk_));
            if (finished_.fetch_add(1, std::memory_order_acq_rel) + 1 == n_chunks) {
                std::lock_guard<std::mutex> lk(mu_);
                done_.notify_one();
            }
        }
    }
    void loop() {
        for (;;) {
            auto fresh = [&] {
                return open(ticket_.load(std::memory_order_acquire)) || stop_.load(std::memory_order_relaxed);
            };
            if (!poll(fresh)) {
                std::unique_lock<std::mutex> lk(mu_);
                cv_.wait(lk, fresh);
            }
            if (stop_.load(std::memory_order_relaxed)) return;
            work();
        }
    }

    static constexpr int kIdxBits = 32;
    static constexpr uint64_t kIdxMask = (1ull << kIdxBits) - 1, kMaxChunks = 1ull << 30;
    const unsigned n_;
    std::vector<std::thread> th_;
    std::mutex mu_;
    std::condition_variable cv_, done_;
    std::atomic<bool> stop_{false};
    void (*call_)(void *, uint64_t, uint64_t) = nullptr;
    void *fn_ = nullptr;
    uint64_t n_job_ = 0, chunk_ = 1;
    std::atomic<uint64_t> ticket_{0}, finished_{0};
};

}  // namespace sg
