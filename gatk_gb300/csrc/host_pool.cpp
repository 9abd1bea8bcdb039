// host_pool.cpp -- see host_pool.h.
#include "host_pool.h"

#include <unistd.h>

#include <algorithm>

namespace ghmm {

namespace {
std::mutex g_mu;
std::shared_ptr<HostPool> g_pool;
int g_refs = 0;
}  // namespace

void HostPool::retain() {
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_refs++ == 0) g_pool.reset(new HostPool());
}

void HostPool::release() {
    std::shared_ptr<HostPool> last;
    std::lock_guard<std::mutex> lk(g_mu);
    if (--g_refs == 0) last.swap(g_pool);
}

std::shared_ptr<HostPool> HostPool::get() {
    std::lock_guard<std::mutex> lk(g_mu);
    return g_pool && g_pool->pid_ == (int)getpid() ? g_pool : nullptr;
}

HostPool::HostPool() : pid_((int)getpid()) {
    const int n = std::max(1, (int)std::thread::hardware_concurrency()) - 1;
    for (int i = 0; i < n; i++) threads_.emplace_back([this] { loop(); });
}

HostPool::~HostPool() {
    if (pid_ != (int)getpid()) {  // the threads exist in the parent process only
        for (auto &t : threads_) t.detach();
        return;
    }
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
    Job job{&work, std::min(helpers, (int)threads_.size())};
    if (job.tickets > 0) {
        {
            std::lock_guard<std::mutex> lk(mu_);
            jobs_.push_back(&job);
        }
        if (job.tickets == 1)
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
