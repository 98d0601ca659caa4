// Host threads for independent pieces of work of one call.
#pragma once

#include <condition_variable>
#include <exception>
#include <mutex>
#include <thread>
#include <type_traits>
#include <vector>

namespace usv {

// Host threads of one solve for the harmonic Ritz steps of its right-hand
// sides: on small grids a cycle takes less GPU time (0.4 ms) than the steps of
// a few right-hand sides one after the other (0.3-0.5 ms each). Started with
// the solve and joined when it returns; a solve of one right-hand side has none.
class HostPool {
  public:
    explicit HostPool(int helpers) {
        try {
            for (int i = 0; i < helpers; ++i) threads_.emplace_back([this] { work(); });
        } catch (const std::exception&) {  // no thread or no memory: those there are and the caller do the work
        }
    }
    ~HostPool() {
        {
            std::lock_guard<std::mutex> l(lock_);
            stop_ = true;
        }
        start_.notify_all();
        for (auto& t : threads_) t.join();
    }
    HostPool(const HostPool&) = delete;
    HostPool& operator=(const HostPool&) = delete;
    // fn(0) .. fn(count - 1), each once, in any order; returns when all are
    // done. fn must not throw.
    template <typename F> void run(int count, F&& fn) {
        if (threads_.empty() || count < 2) {
            for (int i = 0; i < count; ++i) fn(i);
            return;
        }
        auto call = [](void* f, int i) { (*static_cast<std::remove_reference_t<F>*>(f))(i); };
        {
            std::lock_guard<std::mutex> l(lock_);
            call_ = call;
            arg_ = &fn;
            count_ = count;
            next_ = 0;
            left_ = count;
        }
        start_.notify_all();
        drain();
        std::unique_lock<std::mutex> l(lock_);
        done_.wait(l, [this] { return left_ == 0; });
    }

  private:
    void drain() {
        for (;;) {
            int i;
            {
                std::lock_guard<std::mutex> l(lock_);
                if (next_ >= count_) return;
                i = next_++;
            }
            call_(arg_, i);
            std::lock_guard<std::mutex> l(lock_);
            if (--left_ == 0) done_.notify_one();
        }
    }
    void work() {
        for (;;) {
            {
                std::unique_lock<std::mutex> l(lock_);
                start_.wait(l, [this] { return stop_ || next_ < count_; });
                if (stop_) return;
            }
            drain();
        }
    }
    std::vector<std::thread> threads_;
    std::mutex lock_;
    std::condition_variable start_, done_;
    void (*call_)(void*, int) = nullptr;
    void* arg_ = nullptr;
    int count_ = 0, next_ = 0, left_ = 0;
    bool stop_ = false;
};

}  // namespace usv
