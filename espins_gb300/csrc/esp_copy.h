// Host side of the spin transfers: threads that convert between the caller's
// FP64 array and the pinned FP32 ring, chunk by chunk in order, while the
// calling thread issues the copies over the link.
//
// One core converts 11 GB/s of a cold FP64 array, 16 together 140 GB/s, the
// link carries 200 GB/s (FP32): the conversion is the bound.  Starting and
// joining 15 threads for one call takes 300-400 us, so they are kept while any
// handle lives that may use them: one set per process, at most 15, asleep
// between transfers.  Against two alternating FP64 blocks copied by threads of
// each call, set_spins / get_spins into a touched array take: 2.4 MB 179 / 171
// -> 131 / 97 us, 31 MB 886 / 913 -> 342 / 240 us, 403 MB 6.7 / 7.0 -> 3.5 /
// 3.0 ms, 1.36 GB 21.3 / 21.5 -> 12.6 / 10.5 ms.
#pragma once
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace esp {

constexpr int kStageRing = 8;               // chunks in flight, at most
constexpr long long kCopyPiece = 1 << 14;   // values a thread converts at a time

// One transfer of `total` values: value e belongs to chunk e / chunk, staged at
// ring + (chunk number % ring_n) * chunk.  The owner opens chunks (their place
// in the ring is free to be written, or holds the values to read) and waits
// for them, converting pieces itself while it waits: a transfer ends also when
// no other thread helps.
class CopyJob {
public:
    CopyJob(bool to_ring, double *user, float *ring, long long total, long long chunk, int ring_n)
        : to_ring_(to_ring), user_(user), ring_(ring), total_(total), chunk_(chunk), ring_n_(ring_n),
          pieces_((total + kCopyPiece - 1) / kCopyPiece)
    {
        for (std::atomic<int> &d : done_) d.store(0, std::memory_order_relaxed);
    }
    // helpers that a transfer of this size pays for
    int helpers() const { return (int)std::min<long long>(15, total_ / (2 * kCopyPiece)); }
    void open(long long chunks)
    {
        open_.store(std::min(pieces_, chunks * (chunk_ / kCopyPiece)), std::memory_order_release);
    }
    // until every piece of chunk c, which is open, is converted
    void finish(long long c)
    {
        // pieces of this place in the ring up to and with chunk c
        const long long n = std::min(chunk_, total_ - c * chunk_);
        const long long need = c / ring_n_ * (chunk_ / kCopyPiece) + (n + kCopyPiece - 1) / kCopyPiece;
        while (done_[c % ring_n_].load(std::memory_order_acquire) < need) {
            long long p = next_.load(std::memory_order_relaxed);
            if (p < open_.load(std::memory_order_relaxed)) {
                if (next_.compare_exchange_strong(p, p + 1)) convert(p);
            } else {
                std::this_thread::yield();
            }
        }
    }
    // no helper waits for another chunk after this
    void stop() { stop_.store(true, std::memory_order_release); }
    void help()
    {
        for (;;) {
            long long p = next_.load(std::memory_order_relaxed);
            if (p >= pieces_ || stop_.load(std::memory_order_acquire)) return;
            if (p < open_.load(std::memory_order_acquire)) {
                if (next_.compare_exchange_strong(p, p + 1)) convert(p);
            } else {
                std::this_thread::yield();
            }
        }
    }

private:
    void convert(long long p)
    {
        const long long e0 = p * kCopyPiece, c = e0 / chunk_, n = std::min(kCopyPiece, total_ - e0);
        float *f = ring_ + (c % ring_n_) * chunk_ + (e0 - c * chunk_);
        double *d = user_ + e0;
        if (to_ring_)
            for (long long i = 0; i < n; ++i) f[i] = (float)d[i];
        else
            for (long long i = 0; i < n; ++i) d[i] = (double)f[i];
        done_[c % ring_n_].fetch_add(1, std::memory_order_release);
    }
    const bool to_ring_;
    double *user_;
    float *ring_;
    const long long total_, chunk_;
    const int ring_n_;
    const long long pieces_;
    alignas(128) std::atomic<int> done_[kStageRing];
    alignas(128) std::atomic<long long> next_{0};
    alignas(128) std::atomic<long long> open_{0};
    std::atomic<bool> stop_{false};
};

// The threads, shared by the handles of a process; a job is served by those
// that are free.
class CopyPool {
public:
    // the pool that lives while a handle holds it
    static std::shared_ptr<CopyPool> get()
    {
        static std::mutex m;
        static std::weak_ptr<CopyPool> w;
        std::lock_guard<std::mutex> l(m);
        std::shared_ptr<CopyPool> p = w.lock();
        if (!p) w = p = std::make_shared<CopyPool>();
        return p;
    }
    ~CopyPool()
    {
        {
            std::lock_guard<std::mutex> l(m_);
            quit_ = true;
        }
        work_.notify_all();
        for (std::thread &t : threads_) t.join();
    }
    void add(CopyJob &j) noexcept
    {
        const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
        const size_t want = (size_t)std::min(j.helpers(), (int)std::min(16u, hw) - 1);
        if (!want) return;
        std::unique_lock<std::mutex> l(m_);
        try {
            jobs_.push_back({&j, (int)want, 0});
            while (threads_.size() < want) threads_.emplace_back([this] { loop(); });
        } catch (...) {
            // fewer helpers: those there are and the calling thread do the rest
        }
        l.unlock();
        work_.notify_all();
    }
    // takes the job back: no thread uses it afterwards
    void remove(CopyJob &j)
    {
        j.stop();
        std::unique_lock<std::mutex> l(m_);
        const auto here = [&] {
            return std::find_if(jobs_.begin(), jobs_.end(), [&](const Entry &e) { return e.job == &j; });
        };
        if (here() == jobs_.end()) return;
        here()->room = 0;
        idle_.wait(l, [&] { return here()->users == 0; });
        jobs_.erase(here());
    }

private:
    struct Entry {
        CopyJob *job;
        int room, users;   // threads that may still join it, that are in it
    };
    void loop()
    {
        std::unique_lock<std::mutex> l(m_);
        for (;;) {
            auto e = std::find_if(jobs_.begin(), jobs_.end(), [](const Entry &x) { return x.room > 0; });
            if (e == jobs_.end()) {
                if (quit_) return;
                work_.wait(l);
                continue;
            }
            CopyJob *j = e->job;
            --e->room;
            ++e->users;
            l.unlock();
            j->help();
            l.lock();
            e = std::find_if(jobs_.begin(), jobs_.end(), [&](const Entry &x) { return x.job == j; });
            if (--e->users == 0) idle_.notify_all();
        }
    }
    std::mutex m_;
    std::condition_variable work_, idle_;
    std::vector<Entry> jobs_;
    std::vector<std::thread> threads_;
    bool quit_ = false;
};

// A job in the pool for the length of a scope.
class CopyTeam {
public:
    CopyTeam(CopyPool *pool, CopyJob &job) : pool_(pool), job_(job)
    {
        if (pool_) pool_->add(job_);
    }
    ~CopyTeam()
    {
        if (pool_) pool_->remove(job_);
    }
    CopyTeam(const CopyTeam &) = delete;
    CopyTeam &operator=(const CopyTeam &) = delete;

private:
    CopyPool *pool_;
    CopyJob &job_;
};

}  // namespace esp
