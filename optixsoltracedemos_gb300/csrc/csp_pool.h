// csp_pool.h -- host threads of one handle.
#pragma once

#include <condition_variable>
#include <cstddef>
#include <cstdint>
#include <exception>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

namespace csp {

// Host threads for the parallel part of a scene's set-up (element records in ranges), owned by one
// handle, batch or server and joined with it.  run() executes body(k) for k in [0, tasks) on the pool and
// the calling thread and returns when all are done; concurrent callers take turns.  body must not throw.
class HostPool {
public:
    ~HostPool() { stop(); }
    // At least `threads` threads, or as many as the system gives: run() does without any.  One costs about
    // 55 us, so callers ask for what their tasks can use.
    void start(unsigned threads) {
        try {
            th_.reserve(threads);
            while (th_.size() < threads) th_.emplace_back([this] { loop(); });
        } catch (const std::exception&) {  // no thread, or no memory for one
        }
    }
    void stop() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            quit_ = true;
        }
        cv_.notify_all();
        for (auto& t : th_) t.join();
        th_.clear();
        quit_ = false;
    }
    void run(size_t tasks, const std::function<void(size_t)>& body) {
        std::lock_guard<std::mutex> turn(run_mu_);
        {
            std::lock_guard<std::mutex> lk(mu_);
            body_ = &body;
            tasks_ = tasks;
            next_ = 0;
            left_ = tasks;
            ++gen_;
        }
        cv_.notify_all();
        work();
        std::unique_lock<std::mutex> lk(mu_);
        cv_done_.wait(lk, [&] { return left_ == 0; });
        body_ = nullptr;
    }

private:
    // take tasks of the current job until none is left
    void work() {
        for (;;) {
            size_t k;
            const std::function<void(size_t)>* body;
            {
                std::lock_guard<std::mutex> lk(mu_);
                if (!body_ || next_ >= tasks_) return;
                k = next_++;
                body = body_;
            }
            (*body)(k);
            std::lock_guard<std::mutex> lk(mu_);
            if (--left_ == 0) cv_done_.notify_all();
        }
    }
    void loop() {
        uint64_t seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> lk(mu_);
                cv_.wait(lk, [&] { return quit_ || gen_ != seen; });
                if (quit_) return;
                seen = gen_;
            }
            work();
        }
    }
    std::mutex mu_, run_mu_;
    std::condition_variable cv_, cv_done_;
    std::vector<std::thread> th_;
    const std::function<void(size_t)>* body_ = nullptr;
    size_t tasks_ = 0, next_ = 0, left_ = 0;
    uint64_t gen_ = 0;
    bool quit_ = false;
};

}  // namespace csp
