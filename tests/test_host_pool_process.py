"""The host threads' pool by itself, in small programs built from host_pool.cpp: what a process that forks, ends or has
few threads to give does with it."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "gatk_gb300", "csrc")

HEAD = r"""
#include <sys/wait.h>
#include <unistd.h>

#include <atomic>
#include <cstdio>
#include <csignal>
#include <cstdlib>
#include <thread>

#include "host_pool.h"

using ghmm::HostPool;

// the exit status of a child that runs f, -1 when it has not ended after five seconds
template <typename F>
int child(F f) {
    fflush(nullptr);
    const pid_t pid = fork();
    if (pid == 0) {
        f();
        exit(0);
    }
    for (int i = 0; i < 5000; i++) {
        int status = 0;
        if (waitpid(pid, &status, WNOHANG) == pid) return WIFEXITED(status) ? WEXITSTATUS(status) : -2;
        usleep(1000);
    }
    kill(pid, 9);
    waitpid(pid, nullptr, 0);
    return -1;
}
// 0 when a loop over the pool, or on the calling thread where there is none, does all of its work
int loop() {
    std::atomic<int> next{0}, done{0};
    const std::function<void()> work = [&] {
        while (next.fetch_add(1) < 1000) done++;
    };
    if (const auto pool = HostPool::get())
        pool->run(3, work);
    else
        work();
    return done.load() == 1000 ? 0 : 7;
}
"""


def _run(tmp_path, main, flags=(), timeout=120):
    src, exe = tmp_path / "prog.cpp", tmp_path / "prog"
    src.write_text(HEAD + main)
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-pthread", *flags, "-I", CSRC, str(src),
                    os.path.join(CSRC, "host_pool.cpp"), "-o", str(exe)], check=True, capture_output=True)
    return subprocess.run([str(exe)], capture_output=True, text=True, timeout=timeout)


@pytest.mark.parametrize("ends", ["", "HostPool::release();", "HostPool::release(); HostPool::release();",
                                  "if (HostPool::get()) exit(8); if (loop()) exit(9);"])
def test_forked_child_ends(tmp_path, ends):
    """A child of a process with an open pool, whose threads sleep, ends by exit(), also after giving the pool up."""
    r = _run(tmp_path, "int main() { HostPool::retain(4); loop(); usleep(20000); const int rc = child([] { %s });"
                       "printf(\"%%d\", rc); return loop(); }" % ends)
    assert (r.returncode, r.stdout) == (0, "0")


def test_child_forked_while_the_pool_is_in_use(tmp_path):
    """Another thread may hold any of the pool's locks at the moment of the fork."""
    r = _run(tmp_path, r"""
int main() {
    std::atomic<bool> stop{false};
    std::thread other([&] { while (!stop) { HostPool::retain(4); loop(); HostPool::release(); } });
    std::thread third([&] { while (!stop) HostPool::get(); });
    int bad = 0;
    for (int i = 0; i < 200 && !bad; i++) bad = child([] { HostPool::get(); if (loop()) exit(9); });
    stop = true;
    other.join();
    third.join();
    printf("%d", bad);
    return 0;
}""")
    assert (r.returncode, r.stdout) == (0, "0")


def test_process_ends_with_the_pool_open(tmp_path):
    r = _run(tmp_path, "int main() { HostPool::retain(4); return loop(); }")
    assert r.returncode == 0


THREADS = r"""
int main() {
    HostPool::retain(4);
    std::atomic<int> bad{0};
    const std::function<void()> user = [&] { for (int i = 0; i < 300; i++) bad += loop(); };
    std::thread a(user), b(user);
    user();
    a.join();
    b.join();
    HostPool::release();
    return bad.load();
}"""


def test_loops_of_several_threads_have_no_data_race(tmp_path):
    """ThreadSanitizer over loops of three threads at once (where the compiler's runs on this machine)."""
    probe = tmp_path / "probe.cpp"
    probe.write_text("int main() {}")
    exe = str(tmp_path / "probe")
    if subprocess.run([os.environ.get("CXX", "g++"), "-fsanitize=thread", str(probe), "-o", exe],
                      capture_output=True).returncode or subprocess.run([exe], capture_output=True).returncode:
        pytest.skip("no ThreadSanitizer")
    r = _run(tmp_path, THREADS, flags=("-fsanitize=thread", "-g"))
    assert r.returncode == 0 and "data race" not in r.stderr, r.stderr[:2000]


def test_threads_are_those_the_contexts_ask_for(tmp_path):
    r = _run(tmp_path, r"""
#include <filesystem>
int tasks() {
    int n = 0;
    for (const auto &e : std::filesystem::directory_iterator("/proc/self/task")) n += e.exists();
    return n;
}
int main() {
    int bad = 0;
    HostPool::retain(1);
    printf("%d ", tasks());
    bad += loop();
    HostPool::retain(3);
    printf("%d ", tasks());
    bad += loop();
    HostPool::retain(2);
    printf("%d ", tasks());
    for (int i = 0; i < 3; i++) HostPool::release();
    printf("%d", tasks());
    return bad;
}""")
    assert (r.returncode, r.stdout) == (0, "1 3 3 1")


def test_threads_that_cannot_be_started(tmp_path):
    """An address space with room for two or three stacks: the loops run on the threads there are."""
    r = _run(tmp_path, r"""
#include <sys/resource.h>
int main() {
    rlimit stack{}, lim{};
    getrlimit(RLIMIT_STACK, &stack);  // the size of a thread's stack
    long pages = 0;
    FILE *f = fopen("/proc/self/statm", "r");
    if (stack.rlim_cur > ((rlim_t)1 << 30) || !f || fscanf(f, "%ld", &pages) != 1) return 77;
    getrlimit(RLIMIT_AS, &lim);
    lim.rlim_cur = (rlim_t)pages * sysconf(_SC_PAGESIZE) + 3 * stack.rlim_cur;
    setrlimit(RLIMIT_AS, &lim);
    HostPool::retain(64);
    int bad = loop();
    HostPool::release();
    return bad;
}""")
    if r.returncode == 77:
        pytest.skip("no limit on a thread's stack")
    assert r.returncode == 0
