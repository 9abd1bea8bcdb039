// host_pool.cpp -- see host_pool.h.
#include "host_pool.h"

#include <pthread.h>

#include <algorithm>
#include <system_error>

namespace ghmm {

namespace {
// The process's pool.  Never destroyed itself: at exit the threads may still sleep in the pool.
struct Shared {
    std::mutex mu;
    std::shared_ptr<HostPool> pool;
    int refs = 0;
};
Shared *g_shared = new Shared;

// In a forked child the pool's threads do not exist: its mutexes may be held, and its condition variables have waiters,
// for good, so destroying them would wait for ever.  The child leaves all of it as it is and starts without a pool.
void abandon_in_child() { g_shared = new Shared; }
[[maybe_unused]] const int g_registered = pthread_atfork(nullptr, nullptr, abandon_in_child);
}  // namespace

void HostPool::retain(int threads) {
    std::lock_guard<std::mutex> lk(g_shared->mu);
    if (!g_shared->pool) g_shared->pool.reset(new HostPool());
    g_shared->refs++;
    g_shared->pool->grow(threads - 1);
}

void HostPool::release() {
    std::shared_ptr<HostPool> last;
    std::lock_guard<std::mutex> lk(g_shared->mu);
    if (g_shared->refs > 0 && --g_shared->refs == 0) last.swap(g_shared->pool);  // (0: a context of the parent process)
}

std::shared_ptr<HostPool> HostPool::get() {
    std::lock_guard<std::mutex> lk(g_shared->mu);
    return g_shared->pool;
}

void HostPool::grow(int n) {
    std::lock_guard<std::mutex> lk(mu_);
    try {
        while ((int)threads_.size() < n) threads_.emplace_back([this] { loop(); });
    } catch (const std::system_error &) {  // no more threads to be had: the loops run on those there are
    }
}

HostPool::~HostPool() {
    {
        std::lock_guard<std::mutex> lk(mu_);
        stop_ = true;
    }
    wake_.notify_all();
    for (auto &t : threads_) t.join();
}

void HostPool::loop() {
    std::unique_lock<std::mutex> lk(mu_);
    for (;;) {
        wake_.wait(lk, [this] { return stop_ || !jobs_.empty(); });
        if (jobs_.empty()) return;  // stop_
        Job *job = jobs_.front();
        if (--job->tickets == 0) jobs_.pop_front();
        ++job->active;
        lk.unlock();
        (*job->work)();
        lk.lock();
        if (--job->active == 0) done_.notify_all();
    }
}

void HostPool::run(int helpers, const std::function<void()> &work) {
    int tickets;  // (job's go down as helpers join)
    Job job{&work, 0};
    {
        std::lock_guard<std::mutex> lk(mu_);
        job.tickets = tickets = std::min(helpers, (int)threads_.size());
        if (tickets > 0) jobs_.push_back(&job);
    }
    if (tickets > 0) {
        if (tickets == 1)
            wake_.notify_one();
        else
            wake_.notify_all();
    }
    struct Finish {  // also when work() throws: no helper may outlive the job
        HostPool &pool;
        Job &job;
        ~Finish() {
            std::unique_lock<std::mutex> lk(pool.mu_);
            const auto it = std::find(pool.jobs_.begin(), pool.jobs_.end(), &job);
            if (it != pool.jobs_.end()) pool.jobs_.erase(it);
            pool.done_.wait(lk, [this] { return job.active == 0; });
        }
    } finish{*this, job};
    work();
}

}  // namespace ghmm
