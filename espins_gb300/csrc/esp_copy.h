// Host side of the spin transfers: threads that convert between the caller's
// FP64 array and the pinned FP32 ring, chunk by chunk in order, while the
// calling thread issues the copies over the link.
//
// One core converts 11 GB/s of a cold FP64 array, 16 together 140 GB/s, the
// link carries 200 GB/s (FP32): the conversion is the bound.  Starting and
// joining 15 threads for one call takes 300-400 us, so they are kept between
// transfers, asleep.  Against two alternating FP64 blocks copied by threads of
// each call, set_spins / get_spins into a touched array take: 2.4 MB 179 / 171
// -> 131 / 97 us, 31 MB 886 / 913 -> 342 / 240 us, 403 MB 6.7 / 7.0 -> 3.5 /
// 3.0 ms, 1.36 GB 21.3 / 21.5 -> 12.6 / 10.5 ms.
#pragma once
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <list>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include <unistd.h>

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
    static int helpers(long long total) { return (int)std::min<long long>(15, total / (2 * kCopyPiece)); }
    int helpers() const { return helpers(total_); }
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
// that are free.  At most 15, started one by another while their users go on,
// and given back when they have had nothing to do for some seconds or the
// library is unloaded: a program that opens one handle after another starts
// and joins none of them for each.
class CopyPool {
public:
    explicit CopyPool(std::chrono::milliseconds idle = std::chrono::seconds(5))
        : idle_(idle), pid_(getpid()), most_(std::min(16u, std::max(1u, std::thread::hardware_concurrency())) - 1)
    {
    }
    // the process's pool, or null
    static CopyPool *get() noexcept
    {
        // never destroyed, so that it outlives whoever still asks for it; its
        // threads are joined at exit
        static CopyPool *const pool = new (std::nothrow) CopyPool;
        struct AtExit {
            ~AtExit()
            {
                if (pool) pool->close();
            }
        };
        static AtExit at_exit;
        return pool;
    }
    ~CopyPool() { close(); }
    // starts the threads that transfers of this size will use
    void reserve(long long total) noexcept
    {
        if (getpid() != pid_) return;
        std::unique_lock<std::mutex> l(m_);
        grow(l, CopyJob::helpers(total));
    }
    void add(CopyJob &j) noexcept
    {
        const int want = std::min(j.helpers(), (int)most_);
        if (!want || getpid() != pid_) return;   // (a forked child has none of the threads)
        std::unique_lock<std::mutex> l(m_);
        try {
            jobs_.push_back({&j, want, 0});
        } catch (...) {
            return;   // the calling thread does it all
        }
        grow(l, want);
        l.unlock();
        work_.notify_all();
    }
    // takes the job back: no thread uses it afterwards
    void remove(CopyJob &j)
    {
        j.stop();
        if (getpid() != pid_) return;
        std::unique_lock<std::mutex> l(m_);
        const auto here = [&] {
            return std::find_if(jobs_.begin(), jobs_.end(), [&](const Entry &e) { return e.job == &j; });
        };
        if (here() == jobs_.end()) return;
        here()->room = 0;
        idle_users_.wait(l, [&] { return here()->users == 0; });
        jobs_.erase(here());
    }
    // no threads from here on
    void close() noexcept
    {
        if (getpid() != pid_) {
            // a forked child's copies of the handles stand for no threads
            for (std::thread &t : threads_) t.detach();
            for (std::thread &t : done_) t.detach();
            return;
        }
        std::unique_lock<std::mutex> l(m_);
        quit_ = true;
        work_.notify_all();
        left_.wait(l, [&] { return threads_.empty() && !starting_; });
        reap(l);
    }

private:
    struct Entry {
        CopyJob *job;
        int room, users;   // threads that may still join it, that are in it
    };
    // sees to it that there will be `want` threads: starts one, which starts the next
    void grow(std::unique_lock<std::mutex> &l, int want) noexcept
    {
        want_ = std::max(want_, std::min(want, (int)most_));
        reap(l);
        start(l);
    }
    void start(std::unique_lock<std::mutex> &l) noexcept
    {
        if (quit_ || starting_ || (int)threads_.size() >= want_) return;
        starting_ = true;
        l.unlock();
        std::list<std::thread> one;
        try {
            one.emplace_back();
            const auto self = one.begin();
            one.front() = std::thread([this, self] { loop(self); });
        } catch (...) {
            one.clear();   // fewer helpers: those there are and the calling threads do the rest
        }
        l.lock();
        starting_ = false;
        if (one.empty()) want_ = (int)threads_.size();
        threads_.splice(threads_.end(), one);
        started_.notify_all();
        left_.notify_all();
    }
    // joins the threads that have left
    void reap(std::unique_lock<std::mutex> &l) noexcept
    {
        if (done_.empty()) return;
        std::list<std::thread> gone;
        gone.swap(done_);
        l.unlock();
        for (std::thread &t : gone) t.join();
        l.lock();
    }
    void loop(std::list<std::thread>::iterator self) noexcept
    {
        std::unique_lock<std::mutex> l(m_);
        started_.wait(l, [&] { return !starting_; });   // in threads_
        start(l);
        for (;;) {
            auto e = std::find_if(jobs_.begin(), jobs_.end(), [](const Entry &x) { return x.room > 0; });
            if (e == jobs_.end()) {
                if (quit_ || work_.wait_for(l, idle_) == std::cv_status::timeout) {
                    if (!quit_ && std::any_of(jobs_.begin(), jobs_.end(), [](const Entry &x) { return x.room > 0; })) continue;
                    want_ = std::min(want_, (int)threads_.size() - 1);
                    done_.splice(done_.end(), threads_, self);
                    left_.notify_all();
                    return;
                }
                continue;
            }
            CopyJob *j = e->job;
            --e->room;
            ++e->users;
            l.unlock();
            j->help();
            l.lock();
            e = std::find_if(jobs_.begin(), jobs_.end(), [&](const Entry &x) { return x.job == j; });
            if (--e->users == 0) idle_users_.notify_all();
        }
    }
    const std::chrono::milliseconds idle_;
    const pid_t pid_;
    const unsigned most_;
    std::mutex m_;
    std::condition_variable work_, idle_users_, started_, left_;
    std::vector<Entry> jobs_;
    std::list<std::thread> threads_, done_;   // that serve jobs, that have left
    int want_ = 0;
    bool starting_ = false, quit_ = false;
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
