// A few host threads for the work the entry points do beside the device: copies between the caller's pageable memory and
// pinned staging (one thread copies at about 10 GB/s, PCIe takes 55), score sort + NMS of several images. A pool belongs to
// one context or net, is started when that first has enough work for it, sleeps between jobs and ends with its owner. Driven by
// one thread at a time, like its owner.
#pragma once
#include <sched.h>
#include <algorithm>
#include <atomic>
#include <cmath>
#include <condition_variable>
#include <cstdlib>
#include <exception>
#include <fstream>
#include <functional>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

namespace msnh {

// Starts fn(0) .. fn(n - 1) on a thread each, as far as the process may start threads; returns how many did.
template <typename F> int start_threads(std::vector<std::thread> &threads, int n, F fn) {
    int started = 0;
    try {
        threads.reserve(threads.size() + static_cast<size_t>(std::max(0, n)));
        for (; started < n; ++started) threads.emplace_back(fn, started);
    } catch (const std::exception &) {}                       // std::system_error: no more threads; std::bad_alloc
    return started;
}
// fn(0) .. fn(n - 1) shared out over `threads` threads (the caller is one of them); fn must not throw.
template <typename F> void strided_rows(int n, int threads, F &&fn) {
    auto share = [&](int t) { for (int i = t; i < n; i += threads) fn(i); };
    std::vector<std::thread> others;
    const int started = start_threads(others, threads - 1, share);
    for (int t = started; t < threads; ++t) share(t);         // the caller's own, and those that no thread took
    for (auto &th : others) th.join();
}

// The cpus whose time the control groups of this process grant it (rounded up; 0: no limit): the least along the way from its
// group to the root, in the unified hierarchy (cpu.max) and in the cpu controller's own (cpu.cfs_quota_us).
inline int cpu_quota(const std::string &groups = "/proc/self/cgroup", const std::string &root = "/sys/fs/cgroup") {
    double least = 0;
    auto limit = [&](double quota, double period) {
        if (quota > 0 && period > 0 && (least == 0 || quota / period < least)) least = quota / period;
    };
    std::ifstream in(groups);
    std::string line;
    while (std::getline(in, line)) {                          // hierarchy : controllers : path
        const size_t a = line.find(':'), b = a == std::string::npos ? a : line.find(':', a + 1);
        if (b == std::string::npos) continue;
        const std::string controllers = line.substr(a + 1, b - a - 1);
        if (!controllers.empty() && ("," + controllers + ",").find(",cpu,") == std::string::npos) continue;
        const std::string mount = root + (controllers.empty() ? "" : "/" + controllers);
        for (std::string path = line.substr(b + 1);; path.erase(path.find_last_of('/'))) {
            const std::string dir = mount + (path == "/" ? "" : path);
            std::string quota;
            double period = 0, us = 0;
            if (controllers.empty()) {
                std::ifstream f(dir + "/cpu.max");
                if (f >> quota >> period && quota != "max") limit(std::atof(quota.c_str()), period);
            } else {
                std::ifstream q(dir + "/cpu.cfs_quota_us"), p(dir + "/cpu.cfs_period_us");
                if (q >> us && p >> period) limit(us, period);          // (-1: none)
            }
            if (path.find('/') == std::string::npos) break;
        }
    }
    return static_cast<int>(std::ceil(least));
}

class HostPool {
public:
    // threads besides the caller: half of the cpus this process may use (the other half are the same cores' second threads), no
    // more than its control group grants the time of, seven at most (eight copying threads fill PCIe)
    static int default_workers() {
        static const int workers = []() {
            cpu_set_t set;
            int cpus = static_cast<int>(std::thread::hardware_concurrency());
            if (sched_getaffinity(0, sizeof(set), &set) == 0) cpus = CPU_COUNT(&set);
            return workers_for(cpus, cpu_quota());
        }();
        return workers;
    }
    static int workers_for(int cpus, int quota) { return std::max(0, std::min({7, cpus / 2 - 1, quota > 0 ? quota - 1 : 7})); }
    // Where the process may start no more threads the pool makes do with those that started, none of them if need be: the caller
    // takes part in every job.
    explicit HostPool(int workers) {
        start_threads(threads_, workers, [this](int) { work(); });
    }
    int workers() const { return static_cast<int>(threads_.size()); }
    ~HostPool() {
        { std::lock_guard<std::mutex> g(m_); stop_ = true; }
        wake_.notify_all();
        for (auto &t : threads_) t.join();
    }
    HostPool(const HostPool &) = delete;
    HostPool &operator=(const HostPool &) = delete;

    // Starts fn(0) .. fn(n - 1) (fn must not throw). The caller takes part through help() / finish() and has to call finish().
    void begin(int n, std::function<void(int)> fn) {
        std::unique_lock<std::mutex> g(m_);
        idle_.wait(g, [&]() { return active_ == 0; });       // a worker that woke late for the job before
        if (static_cast<int>(done_size_) < n) { done_.reset(new std::atomic<bool>[n]); done_size_ = n; }
        fn_ = std::move(fn); n_ = n;
        for (int i = 0; i < n; ++i) done_[i].store(false, std::memory_order_relaxed);
        next_.store(0, std::memory_order_relaxed);
        ++job_;
        g.unlock();
        wake_.notify_all();
    }
    bool help(int below = 0x7fffffff) {                       // one item (one before `below`) on the calling thread; false: none left to start
        int i = next_.load(std::memory_order_relaxed);
        do { if (i >= n_ || i >= below) return false; } while (!next_.compare_exchange_weak(i, i + 1, std::memory_order_acq_rel, std::memory_order_relaxed));
        fn_(i);
        done_[i].store(true, std::memory_order_release);
        return true;
    }
    bool all_started(int below) const { return next_.load(std::memory_order_relaxed) >= std::min(below, n_); }   // (of the items before `below`)
    bool done(int i) const { return done_[i].load(std::memory_order_acquire); }
    void finish() {
        while (help()) {}
        for (int i = 0; i < n_; ++i) while (!done(i)) std::this_thread::yield();
    }
    void run(int n, std::function<void(int)> fn) { begin(n, std::move(fn)); finish(); }

private:
    void work() {
        unsigned long seen = 0;
        std::unique_lock<std::mutex> g(m_);
        while (true) {
            wake_.wait(g, [&]() { return stop_ || job_ != seen; });
            if (stop_) return;
            seen = job_;
            ++active_;
            g.unlock();
            while (help()) {}
            g.lock();
            if (--active_ == 0) idle_.notify_all();
        }
    }
    std::mutex m_;
    std::condition_variable wake_, idle_;
    std::vector<std::thread> threads_;
    std::function<void(int)> fn_;
    std::unique_ptr<std::atomic<bool>[]> done_;
    size_t done_size_ = 0;
    int n_ = 0, active_ = 0;
    std::atomic<int> next_{0};
    unsigned long job_ = 0;
    bool stop_ = false;
};

}  // namespace msnh
