// host_pool.h -- the worker threads that the host loops of a process's contexts share.  Starting threads for every
// loop cost about 0.13 ms a thread on the GB300 hosts' Arm cores: a call of one region, with three loops, took 2.0 ms,
// with the pool 0.43.
#pragma once

#include <condition_variable>
#include <deque>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace ghmm {

class HostPool {
public:
    // One reference per open context (ghmm_initialize / ghmm_done), with the threads its loops may run on, the caller's
    // one of them: the pool has as many as the context with the most asks for (or as could be started) until the last
    // reference goes.
    static void retain(int threads);
    static void release();
    // The live pool, or null: no context of this process is open (a forked child starts without the parent's).
    static std::shared_ptr<HostPool> get();

    // work() on the calling thread and on up to `helpers` pool threads at once; returns when all of them have returned.
    // Several threads may call it at the same time.  A helper that is busy elsewhere until the caller's own work()
    // returns does not join any more, so work() must be a loop over a shared cursor.
    void run(int helpers, const std::function<void()> &work);

    ~HostPool();

private:
    struct Job {
        const std::function<void()> *work;
        int tickets;     // helpers that may still join
        int active = 0;  // helpers inside work()
    };
    HostPool() = default;
    void grow(int n);
    void loop();

    std::mutex mu_;
    std::condition_variable wake_, done_;
    std::deque<Job *> jobs_;
    std::vector<std::thread> threads_;
    bool stop_ = false;
};

}  // namespace ghmm
