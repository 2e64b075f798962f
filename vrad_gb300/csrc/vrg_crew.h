// vrg_crew.h -- host threads that end with the scope they serve.
#pragma once

#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace vrg {

// Tasks on threads of their own, or on the caller's where no thread can be had.
// What a task throws waits for join(); an exception that left its thread
// would end the process.
class Crew {
public:
    Crew() = default;
    Crew(const Crew &) = delete;
    Crew &operator=(const Crew &) = delete;
    ~Crew() { wait(); }

    template <class F>
    void run(F f) {
        auto task = [this, f] {
            try {
                f();
            } catch (...) {
                std::lock_guard<std::mutex> lk(mu_);
                if (!error_) error_ = std::current_exception();
            }
        };
        try {
            pool_.emplace_back(task);
        } catch (...) {
            task();
        }
    }

    // Waits for the tasks, then throws what the first failed one threw.
    void join() {
        wait();
        if (error_) std::rethrow_exception(error_);
    }

private:
    void wait() {
        for (std::thread &t : pool_) t.join();
        pool_.clear();
    }

    std::vector<std::thread> pool_;
    std::mutex mu_;
    std::exception_ptr error_;
};

}  // namespace vrg
